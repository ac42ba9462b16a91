// Host-only harness for the rules of the chunked decoder that need no GPU (plan.h).
#include <stddef.h>
#include <stdint.h>

#include "plan.h"

extern "C" uint32_t mmr_test_slice_share(uint32_t n, uint32_t base, uint32_t blocks, uint32_t si, uint32_t sched_len) {
    return mmr::slice_share(n, base, blocks, si, sched_len);
}
