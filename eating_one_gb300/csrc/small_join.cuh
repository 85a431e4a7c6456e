// small_join.cuh - joins of build sides that fit in shared memory (small_join.cu).
#pragma once

#include "ej_internal.h"

// True when a hash join or left outer join on nR build rows takes the
// shared-memory join: at most BT_ROWS (16384) rows, and no option of the
// handle asks for a build, a table format, partition bits, a load factor or a
// probe block shape (a tuning table's entries choose among the tables in
// global memory).  One join into a given output, |S| = 4 |R|, here and with
// the fastest global table: 2^10 rows 48 and 104 us, 2^12 49 and 123, 2^14 54
// and 129.
bool ej_small_join_applies(const ej_handle* h, uint64_t nR);

// rows to out (count_only: none), the count into the device word *cursor
// (zeroed here); outer: one NULL-extended row per S row without a match
ej_status ej_small_join(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS, bool outer,
                        bool count_only, ej_result* out, uint64_t cap, unsigned long long* cursor);
