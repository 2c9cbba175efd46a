// Host build of the hot kernels' point arithmetic (mhd_hot.cuh) for
// tests/test_cpu_hot_args.py.
#include "../beta1_b200/csrc/mhd_hot.cuh"

using namespace mhd;

extern "C" {

// quotients of numerators t[0..n) by d, as the kernels form them
void hot_quot(uint32_t d, const uint32_t *t, uint32_t *q, int n)
{
    const FastDiv f = fast_div(d);
    for (int i = 0; i < n; ++i)
        q[i] = fast_quot(t[i], f);
}

int hot_plane_of(int f) { return plane_of(f); }
}
