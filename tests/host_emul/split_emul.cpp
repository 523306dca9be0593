// The rule that cuts K of a dense linear at decode rows (turboexl3_b200/csrc/t3_split.h), for tests/test_plan_sweep_host.py.
#include "../../turboexl3_b200/csrc/t3_split.h"

// slices of `nb` x `blocks` blocks on `sms` multiprocessors, where shared memory is no limit; + 100: a CTA a multiprocessor
extern "C" int split_emul(unsigned sms, unsigned nb, unsigned blocks) {
    uint32_t alone = 0;
    const uint32_t s = t3::pick_split_dense(sms, nb, blocks, 1u, 1u << 20, 1u << 20, alone, [](uint32_t, uint32_t) { return 0u; });
    return (int)(s + (alone ? 100u : 0u));
}
