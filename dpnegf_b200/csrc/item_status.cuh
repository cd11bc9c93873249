// What a sweep item's status says of the flags that its kernel collected.
#pragma once
#include "../../include/negf_b200.h"

#ifdef __CUDACC__
#define NEGF_HD __host__ __device__
#else
#define NEGF_HD
#endif

// inv_bad: a block inverse failed; inv_lost: one of them because a bounded wait for a panel expired, so that it
// was not stored (the numbers behind it are arbitrary, so this goes before the pivots met in them); tc_lost: a
// bounded tensor-core wait expired; finite: T and DOS are.
NEGF_HD inline int item_status(bool inv_bad, bool inv_lost, bool tc_lost, bool finite) {
  if (inv_bad) return inv_lost ? NEGF_ERR_TIMEOUT : NEGF_ERR_SINGULAR;
  if (tc_lost) return NEGF_ERR_TIMEOUT;
  return finite ? NEGF_OK : NEGF_ERR_NONFINITE;
}
