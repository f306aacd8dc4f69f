// fsg_perturb_bs32.cu -- the Burning Ship family perturbation loop with
// FP32-mantissa + int32-exponent deltas: fsg_bs.cuh instantiated on fr
// (the reference's loop, perturbation.py:1468-1811, in that arithmetic), one
// kernel per flavor so that the closures' flavor branches fold, two for flavor 1
// (references on the real axis), each at two occupancies but for flavor 5.
#include "fsg_bs.cuh"

template <int FL, bool AXIS, bool DENSE>
static void launch_bs_fr(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    const size_t sm = fsg_starts_smem(W) + 4 * sizeof(unsigned long long) * (size_t)block;
    k_perturb_bs<fr, FL, AXIS, DENSE><<<fsg_auto_grid(k_perturb_bs<fr, FL, AXIS, DENSE>, grid, block,
                                                      W.total - W.base, sm), block, sm, s>>>(W, C);
}
template <int FL, bool AXIS>
static void launch_bs_size(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    const size_t sm = fsg_starts_smem(W) + 4 * sizeof(unsigned long long) * 256;
    const long long three = 256LL * fsg_auto_grid(k_perturb_bs<fr, FL, AXIS, false>, 0, 256, 1LL << 40, sm);
    if (W.total - W.base > three) launch_bs_fr<FL, AXIS, true>(W, C, grid, block, s);
    else launch_bs_fr<FL, AXIS, false>(W, C, grid, block, s);
}

void fsg_launch_perturb_bs_fe32(const WorkDev &W, const CalcDev &C, int grid, int block,
                                cudaStream_t s) {
    switch (C.flavor) {
    case 1:
        if (C.axis) launch_bs_size<1, true>(W, C, grid, block, s);
        else launch_bs_size<1, false>(W, C, grid, block, s);
        break;
    case 2: launch_bs_size<2, false>(W, C, grid, block, s); break;
    case 3: launch_bs_size<3, false>(W, C, grid, block, s); break;
    case 4: launch_bs_size<4, false>(W, C, grid, block, s); break;
    default: launch_bs_fr<5, false, false>(W, C, grid, block, s); break;
    }
}
