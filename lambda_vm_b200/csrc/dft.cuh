// One DFT pass over a row-major matrix: its arguments and the root tables,
// shared by the two kernels that run passes (ntt.cu k_dft on the integer
// pipes, ntt_tc.cu k_dft_tc on the tensor cores).
#pragma once
#include "common.cuh"
#include "gl.cuh"

namespace sg {

// omega_N^e = lo[e & (2^h - 1)] * hi[e >> h], N = 2^logN.
struct Tw {
    const uint64_t* lo;
    const uint64_t* hi;
    uint32_t h;
    uint32_t logN;
};

__device__ __forceinline__ uint64_t tw_pow(const Tw& t, uint64_t e) {
    return gl::mul(__ldg(t.lo + (e & ((1ULL << t.h) - 1))), __ldg(t.hi + (e >> t.h)));
}

// omega_{2^logM}^{+-x}
__device__ __forceinline__ uint64_t tw_root(const Tw& t, uint32_t logM, uint64_t x, bool inv) {
    const uint64_t mask = (1ULL << t.logN) - 1;
    uint64_t e = (x << (t.logN - logM)) & mask;
    if (inv) e = (mask + 1 - e) & mask;
    return tw_pow(t, e);
}

struct PassArgs {
    const uint64_t* in;
    uint64_t* out;
    uint64_t m;               // columns transformed
    uint64_t in_ld, out_ld;   // row strides of in / out in u64 (>= m)
    uint32_t logL;
    uint32_t inverse;
    // row(tile, point, rep) = tile*ts + point*ps + rep*rs
    uint64_t in_ts, in_ps;
    uint64_t out_ts, out_ps, out_rs;
    uint32_t reps;
    Tw tw;
    uint32_t pre_kind;   // 0: none, 1: omega_{2^pre_log}^{in_row * rep}
    uint32_t pre_log;
    uint32_t post_kind;  // 0: none, 1: omega_{2^post_log}^{+-(tile*k)}, 2: weights[out_row], 3: scalar
    uint32_t post_log;
    const uint64_t* weights;
    uint64_t scalar;
    uint32_t canon_out;
};

// Points (rows x columns x cosets) of a pass above which k_dft_tc takes it.
constexpr uint64_t TC_MIN_POINTS = 1ULL << 20;

// Whether k_dft_tc runs this pass (its length, kinds and size), and its
// launch; see ntt_tc.cu.
bool dft_tc_takes(const PassArgs& a, uint64_t ntiles);
int launch_dft_tc(Ctx* ctx, cudaStream_t st, const PassArgs& a, uint64_t ntiles);

}  // namespace sg
