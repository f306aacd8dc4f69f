// fsg_perturb_bs64.cu -- the Burning Ship family perturbation loop in the
// reference's two delta forms (perturbation.py:1406-1811 with the closures of
// models/burning_ship.py:19-60, 535-859): fsg_bs.cuh instantiated on double, one
// kernel per flavor so that the closures' flavor branches fold (two for flavor 1:
// references on the real axis have their own), and on float64
// Xrange records (the Xrange branch).
//
// Built with -fmad=false so that every operation rounds once in the order of
// the reference source.
#include "fsg_bs.cuh"

template <class T, int FL, bool AXIS>
static void launch_bs(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    const size_t acc = 4 * sizeof(unsigned long long);      // per thread
    size_t sm = fsg_starts_smem(W);
    block = fsg_fp64_block(k_perturb_bs<T, FL, AXIS, false>, grid, block, W.total - W.base, sm + 256 * acc);
    sm += acc * (size_t)block;
    k_perturb_bs<T, FL, AXIS, false><<<fsg_auto_grid(k_perturb_bs<T, FL, AXIS, false>, grid, block, W.total - W.base, sm),
                          block, sm, s>>>(W, C);
}

void fsg_launch_perturb_bs(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    if (C.mode == 1) { launch_bs<xf, 0, false>(W, C, grid, block, s); return; }
    switch (C.flavor) {
    case 1:
        if (C.axis) launch_bs<double, 1, true>(W, C, grid, block, s);
        else launch_bs<double, 1, false>(W, C, grid, block, s);
        break;
    case 2: launch_bs<double, 2, false>(W, C, grid, block, s); break;
    case 3: launch_bs<double, 3, false>(W, C, grid, block, s); break;
    case 4: launch_bs<double, 4, false>(W, C, grid, block, s); break;
    default: launch_bs<double, 5, false>(W, C, grid, block, s); break;
    }
}
