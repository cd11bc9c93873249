// What a sweep item's status says of the flags that its kernel collected.
#pragma once
#include "../../include/negf_b200.h"

#ifdef __CUDACC__
#define NEGF_HD __host__ __device__
#else
#define NEGF_HD
#endif

// Flags of a block inverse; an item collects those of its blocks.
constexpr int INV_SINGULAR = 1;  // a zero or non-finite pivot
constexpr int INV_LOST = 2;      // a bounded wait for a panel expired: the inverse was not stored

// `inv`: the collected flags; tc_lost: a bounded tensor-core wait expired; finite: T and DOS are.
// A lost inverse leaves arbitrary numbers behind it, so it goes before the pivots met in them.
NEGF_HD inline int item_status(int inv, bool tc_lost, bool finite) {
  if (inv & INV_LOST) return NEGF_ERR_TIMEOUT;
  if (inv) return NEGF_ERR_SINGULAR;
  if (tc_lost) return NEGF_ERR_TIMEOUT;
  return finite ? NEGF_OK : NEGF_ERR_NONFINITE;
}
