// The delta rule's kernels whose walk waits, for a short while, for bytes that never come.
#define TC_WAIT_LIMIT (1u << 14)
#define TC_DRAIN_LIMIT (1u << 14)
#define DP_STRAY 16
#include "delta_rule_parallel.cu"
