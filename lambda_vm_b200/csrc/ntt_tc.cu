// DFT passes on the tensor cores (tcgen05 kind::i8), bit for bit the values of
// ntt.cu's k_dft.
//
// A 2^r-point DFT over Goldilocks is a matrix product with constants, and a
// matrix product mod p is an integer one on bytes: with x = sum_b x_b 2^8b (the
// bytes of the 64-bit word as it lies in memory) and the constant
// w^jk 2^8b mod p = sum_d c_d 2^8d,
//   X_k = sum_d 2^8d * ( sum_{j,b} c_d(k,j,b) x_b(j) )   (mod p),
// so the eight limbs d of every output k are one u8 x u8 -> s32 product of the
// (8 R) x (8 R) byte matrix c with the raw bytes of the R inputs. The sums
// stay below 256 * 255^2 < 2^24, so nothing is rounded; the limbs are put
// together as an 80-bit number and reduced once (11 instructions a point
// where a radix-32 butterfly network in registers takes about 130).
//
// Layout. A pass of L = R1 R2 points (x 2 for L = 2^11, see DBL) runs as two
// such products with the L-point twiddles between them. The kernel is
// persistent, one CTA per SM: 16 working warps and one that issues the
// products. A tile is 16384 points (S columns x T points), held as a 128 KB
// byte matrix A in shared memory in the K-major core-matrix layout the MMA
// reads (8 rows x 16 bytes; rows = DFT instances, K = the inputs' bytes):
//   stage 1: rows (j2, s), K = j1, as M-tiles of 128 rows: tile m holds the
//            j2 of its own share of A;
//   stage 2: rows (k1, s), K = j2: K slices of 16 bytes = two j2 over all
//            rows, so M-tile m's outputs land exactly in the part of A that
//            M-tile m was read from, and the exchange is in place.
// A stage takes four steps of 256 TMEM columns (the products of one M-tile for
// R = 32, two for R = 16, four for R = 8) in two accumulators. The warps meet
// only through mbarriers (product complete, accumulator read, tile landed,
// stage 1's outputs written), so the products run under the arithmetic and the warps
// drift apart; the next tile's loads (8-byte asynchronous copies: the bytes
// of a word stay together, the words of a row segment go to different rows)
// start when stage 2's last product has completed, under its last two steps.
// The constant matrix (64 KB for R = 32) is written to shared memory by the
// CTA itself when it starts.
//
// Measured on the 2^20 x 256, blowup 4 LDE (four passes, ten matrix-sized
// units): k_dft 25.5 ms, this kernel 18.3 ms. With its arithmetic taken out it
// takes 14.3 ms, without its HBM accesses 14.1, with neither 8.6. The products
// run at the tensor cores' full i8 rate (128 cycles per 128 x 256 x 32) and
// take 4.6 ms of it; the arithmetic issues 64 cycles a warp for a stage-1
// output. The HBM side is not bound by bytes (DRAM 20 % busy): a tile's 128 KB
// are asked for in one burst, in its last two steps, as 128-byte row segments
// (16 columns of a 2^10-point tile). 8 columns (two independent groups of 256
// threads) took 18.9 ms, touching the next tile's rows with L2 prefetches on
// top 37.7; scratch matrices in blocks of 16 columns, whole tiles of which are
// contiguous, made no difference (18.35).
//
// Coset shifts cost nothing: a forward pass over coset `rep` multiplies input
// i by w_{B L}^{i rep}; its j1 part goes into the constant matrix, the j2 part
// into the twiddle table and the tile's part into the output factor. A CTA
// therefore works on one rep (grid a multiple of reps), which also brings the
// reps' reads of one input tile together in L2.
//
// No unit is full: 36-47 % of the issue slots (110 thread instructions a point
// and pass where k_dft takes 180-230), 1.8 TB/s of DRAM traffic, the i8 unit a
// quarter of the time. A tile's phases (loads, products, arithmetic) overlap
// too little: 18.3 ms against 14 for the arithmetic or the accesses alone.
#include <type_traits>

#include "common.cuh"
#include "dft.cuh"
#include "gl.cuh"
#include "tc.cuh"

namespace sg {

using namespace tc;

namespace {

constexpr uint32_t NT = 512;                // working threads; one more warp issues the products
constexpr uint32_t PTS = 16384;             // points of a tile
constexpr uint32_t A_BYTES = 8 * PTS;       // the byte matrix
constexpr uint32_t TMEM_COLS = 512;

// Shared-memory plan of one instantiation, in bytes.
template <int LR1, int LR2, bool DBL, bool FLAT>
struct TcPlan {
    static constexpr uint32_t R1 = 1u << LR1, R2 = 1u << LR2, T = R1 * R2, D = DBL ? 2 : 1;
    static constexpr uint32_t S = PTS / T;   // slots: columns (x parity for DBL) of a tile
    static constexpr uint32_t CSL = S / D;   // columns of a tile
    static constexpr uint32_t B1 = 64 * R1 * R1, B2 = R1 == R2 ? 0 : 64 * R2 * R2;
    static constexpr uint32_t AB = FLAT ? CSL * (R1 + D * R2) : R1 + D * R2;  // factor words a, b
    static constexpr uint32_t X_WORDS = FLAT ? AB : T + 2 * AB;
    static constexpr uint32_t OFF_B2 = R1 == R2 ? 0 : B1;
    static constexpr uint32_t OFF_A = B1 + B2;
    static constexpr uint32_t OFF_TW = OFF_A + A_BYTES;
    static constexpr uint32_t OFF_X = OFF_TW + 8 * T;
    static constexpr uint32_t OFF_W = OFF_X + 8 * X_WORDS;
    static constexpr uint32_t OFF_BAR = OFF_W + (DBL ? 8 * T : 0);
    static constexpr uint32_t SMEM = OFF_BAR + 64;
    static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
};

// One step's products: MT accumulators of 128 x N s32 side by side from TMEM
// column d on = A (128 rows each, A_TILE bytes apart) x B (N rows)^T over
// KS K steps of 32 bytes, then an arrive on `bar` when they have completed.
// Issued by one elected thread of a converged warp.
template <uint32_t MT, uint32_t N, uint32_t KS, uint32_t A_TILE, uint32_t A_LBO, uint32_t B_LBO>
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t a, uint32_t b, uint32_t bar) {
    if (elect_one()) {
        const uint64_t db = mma_desc(b, B_LBO, 128);
#pragma unroll
        for (uint32_t t = 0; t < MT; ++t) {
            const uint64_t da = mma_desc(a + t * A_TILE, A_LBO, 128);
#pragma unroll
            for (uint32_t k = 0; k < KS; ++k)
                mma_i8(d + t * N, da + k * ((2 * A_LBO) >> 4), db + k * ((2 * B_LBO) >> 4), N, k);
        }
        mma_commit(bar);
    }
    __syncwarp();
}

// 32 accumulator columns of this thread's lane; the registers hold them after tmem_wait.
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {"
        "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31"
        "}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
}
// The loads issued so far have landed; r (the last one's) is an operand, so
// that its uses stay behind the wait.
__device__ __forceinline__ void tmem_wait(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
          "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
          "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
          "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
        :
        : "memory");
}

// The word of the eight limb sums v_d < 2^24: sum_d v_d 2^8d mod p, as an
// 80-bit number of three words (v + 256 v' < 257 * 256 * 255^2 < 2^32).
__device__ __forceinline__ uint64_t recombine(const uint32_t* v) {
    const uint32_t p0 = v[0] + (v[1] << 8), p1 = v[2] + (v[3] << 8), p2 = v[4] + (v[5] << 8), p3 = v[6] + (v[7] << 8);
    uint32_t w0, w1, w2;
    asm("add.cc.u32 %0, %3, %4;\n\t"
        "addc.cc.u32 %1, %5, %6;\n\t"
        "addc.u32 %2, %7, 0;"
        : "=r"(w0), "=r"(w1), "=r"(w2)
        : "r"(p0), "r"(p1 << 16), "r"(p1 >> 16), "r"(p2), "r"(p3 >> 16));
    asm("add.cc.u32 %0, %0, %2;\n\t"
        "addc.u32 %1, %1, 0;"
        : "+r"(w1), "+r"(w2)
        : "r"(p3 << 16));
    return gl::reduce96(w0, w1, w2);
}

// Barrier of the 512 working threads; the OR of their predicates.
__device__ __forceinline__ bool bar_or(bool x) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(ok)
        : "r"((uint32_t)x), "n"(NT)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bar_all() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }
// The byte matrix of an R-point DFT over coset `shift` of 2^lb:
// c(k, j, b) = w_R^{+-jk} w_{2^lb R}^{shift j} 2^8b, at row 8 k + d, K byte
// 8 j + b in the core-matrix layout (K slice stride 128 R bytes).
template <int LR, bool INV>
__device__ void write_matrix(uint8_t* B, const Tw& tw, uint32_t lb, uint32_t shift) {
    constexpr uint32_t R = 1u << LR;
    const uint64_t mask = (1ull << tw.logN) - 1;
    for (uint32_t e = threadIdx.x; e < R * R; e += NT + 32) {
        const uint32_t k = e / R, j = e % R;
        uint64_t x = ((uint64_t)(j * k) << (tw.logN - LR)) & mask;
        if (INV) x = (mask + 1 - x) & mask;
        if (lb) x = (x + ((uint64_t)(shift * j) << (tw.logN - lb - LR))) & mask;
        uint64_t c = gl::canon(tw_pow(tw, x)), row[8];
#pragma unroll
        for (int d = 0; d < 8; ++d) row[d] = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
#pragma unroll
            for (int d = 0; d < 8; ++d) row[d] |= ((c >> (8 * d)) & 0xFF) << (8 * b);
            c = gl::canon(gl::mul_2exp<8>(c));
        }
        const uint32_t at = smem_addr(B) + (j >> 1) * (128 * R) + k * 128 + (j & 1) * 8;
#pragma unroll
        for (int d = 0; d < 8; ++d) sts64(at + d * 16, row[d]);
    }
}

template <int LR1, int LR2, bool DBL, bool INV, bool FLAT, int POST>
__global__ void __launch_bounds__(NT + 32, 1)
    k_dft_tc(PassArgs a, uint32_t gtiles, uint32_t ctiles, uint64_t flat_total, uint32_t lb, unsigned* err) {
    using PL = TcPlan<LR1, LR2, DBL, FLAT>;
    constexpr uint32_t R1 = PL::R1, R2 = PL::R2, T = PL::T, S = PL::S, D = PL::D, CSL = PL::CSL;
    constexpr uint32_t ROWS2 = PTS / R2;  // instances of each stage
    constexpr uint32_t A_WORDS = FLAT ? CSL * R1 : R1;      // factor words a; b follows
    extern __shared__ __align__(1024) uint8_t sm8[];
    const uint32_t tid = threadIdx.x, lane = tid % 32;
    const uint32_t warp = __shfl_sync(0xffffffffu, tid / 32, 0);  // warp-uniform
    const uint32_t rep = blockIdx.x % a.reps;
    uint64_t* TW = reinterpret_cast<uint64_t*>(sm8 + PL::OFF_TW);  // [k1][j2]
    uint64_t* TWX = reinterpret_cast<uint64_t*>(sm8 + PL::OFF_X);  // [k1][j2], with the tile's factor
    uint64_t* FA0 = FLAT ? TWX : TWX + T;                          // tile factors a[k1], b[parity][k2]: two tiles'
    uint64_t* W = reinterpret_cast<uint64_t*>(sm8 + PL::OFF_W);    // DBL: w_2T^i
    // Barriers: an accumulator's product is complete (per accumulator), the 16
    // warps have read it (per accumulator), the tile's inputs have landed, and
    // stage 1's outputs are in A; the last one is for a CTA that gives up.
    const uint32_t bar_full = smem_addr(sm8 + PL::OFF_BAR), bar_read = bar_full + 16, bar_loaded = bar_full + 32,
                   bar_ready = bar_full + 40, bar_drain = bar_full + 56;
    uint32_t* ctrl = reinterpret_cast<uint32_t*>(sm8 + PL::OFF_BAR + 48);  // TMEM address, abort word
    volatile uint32_t* abort = ctrl + 1;
    const uint64_t mask = (1ull << a.tw.logN) - 1;

    // ---- set-up: TMEM, barriers, constant matrices, twiddles
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(ctrl)),
                     "n"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(bar_full, 1), mbar_init(bar_full + 8, 1);
        mbar_init(bar_read, NT / 32), mbar_init(bar_read + 8, NT / 32);
        mbar_init(bar_loaded, NT), mbar_init(bar_ready, NT / 32), mbar_init(bar_drain, 1);
        *abort = 0;
    }
    const uint32_t r2 = R1 == R2 ? rep : 0;  // one matrix serves both stages when R1 == R2
    write_matrix<LR1, INV>(sm8, a.tw, lb, rep);
    if constexpr (R1 != R2) write_matrix<LR2, INV>(sm8 + PL::OFF_B2, a.tw, 0, 0);
    for (uint32_t e = tid; e < T; e += NT + 32) {
        const uint32_t k1 = e / R2, j2 = e % R2;
        uint64_t x = ((uint64_t)(j2 * k1) << (a.tw.logN - LR1 - LR2)) & mask;
        if (INV) x = (mask + 1 - x) & mask;
        if (lb) {
            x += (uint64_t)(rep * j2) << (a.tw.logN - lb - LR1 - LR2);
            x -= (uint64_t)(r2 * j2) << (a.tw.logN - lb - LR2);
            x &= mask;
        }
        TW[e] = tw_pow(a.tw, x);
        if constexpr (DBL) W[e] = tw_root(a.tw, LR1 + LR2 + 1, e, INV);
    }
    // DBL: the second half's input i + T carries w_{2^lb L}^{rep T} = w_{2^lb}^{rep} more than input i
    // (2^lb counts the cosets of the T-point DFTs: twice the pass's own)
    uint64_t gsh = 1;
    if constexpr (DBL)
        if (lb && rep) gsh = tw_root(a.tw, lb, rep, false);
    fence_async();
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = ctrl[0];
    const uint32_t Ab = smem_addr(sm8) + PL::OFF_A, B1 = smem_addr(sm8), B2 = smem_addr(sm8) + PL::OFF_B2;
    const uint32_t t0 = blockIdx.x / a.reps, gstep = gridDim.x / a.reps;
    if (warp == NT / 32) {
        // ---- the issuing warp: every step's products as soon as their inputs
        // are there and their accumulator has been read
        uint32_t uses = 0;  // of each accumulator so far
        auto gave_up = [&] { return __any_sync(0xffffffffu, *abort != 0); };  // one answer for the warp
        for (uint32_t t = t0, n = 0; t < gtiles && !gave_up(); t += gstep, ++n) {
#pragma unroll 1
            for (uint32_t st = 0; st < 2; ++st) {
                mbar_wait(st ? bar_ready : bar_loaded, n & 1, abort, err);
                fence_async();
#pragma unroll 1
                for (uint32_t step = 0; step < 4; ++step) {
                    const uint32_t b = step & 1;
                    if (uses) mbar_wait(bar_read + 8 * b, (uses - 1) & 1, abort, err);
                    tc_after();
                    if (st == 0) {
                        constexpr uint32_t MT = 32 / R1, TILE = 128 * 8 * R1;
                        mma_step<MT, 8 * R1, R1 / 4, TILE, 2048, 128 * R1>(tmem + b * 256, Ab + step * MT * TILE, B1,
                                                                           bar_full + 8 * b);
                    } else {
                        constexpr uint32_t MT = 32 / R2;
                        mma_step<MT, 8 * R2, R2 / 4, 2048, 16 * ROWS2, 128 * R2>(tmem + b * 256, Ab + step * MT * 2048,
                                                                                 B2, bar_full + 8 * b);
                    }
                    if (b) ++uses;
                }
            }
        }
        if (gave_up()) {
            if (elect_one()) mma_commit(bar_drain);
            __syncwarp();
            mbar_drain(bar_drain, 0);
        }
        __syncthreads();
        tc_after();
        return;
    }
    // A stage's four steps: body(step, i, k0, r) gets the 4 outputs k0..k0+3 of
    // instance row i as 32 limb sums, twice a step. With `together` the last
    // two products are waited for at once: A is no longer read when body(2,
    // ...) starts.
    auto stage = [&](auto rc, bool together, auto&& body) {
        constexpr uint32_t R = decltype(rc)::value;
        // a warp's 64 columns: 8 outputs of one of the step's 32 / R M-tiles
        const uint32_t k0 = 8 * ((warp >> 2) % (R / 8)), row0 = 128 * ((warp >> 2) / (R / 8)) + 32 * (warp & 3) + lane;
#pragma unroll 1
        for (uint32_t step = 0; step < 4; ++step) {
            // an accumulator is used four times a tile, so its parities repeat
            if (!(together && step == 3)) mbar_wait(bar_full + 8 * (step & 1), step >> 1, abort, err);
            if (together && step == 2) mbar_wait(bar_full + 8, 1, abort, err);
            tc_after();
            const uint32_t from = tmem + ((32u * (warp & 3)) << 16) + (step & 1) * 256 + 64 * (warp >> 2);
            const uint32_t i = step * (4096 / R) + row0;
            uint32_t r[2][32];
            tmem_ld32(from, r[0]);
            tmem_wait(r[0]);
            tmem_ld32(from + 32, r[1]);
            body(step, i, k0, r[0]);
            tmem_wait(r[1]);
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_read + 8 * (step & 1));
            body(step, i, k0 + 4, r[1]);
        }
    };

    const uint64_t ip = a.in_ps * a.in_ld, op = a.out_ps * a.out_ld;
    const uint32_t m32 = (uint32_t)a.m;
    // flat tiles: slot column c of tile t is column (t CSL + c) of the ntiles x m grid of columns
    auto locate = [&](uint32_t t, uint32_t c, uint32_t& pt, uint32_t& col) -> bool {
        if constexpr (FLAT) {
            const uint64_t f = (uint64_t)t * CSL + c;
            pt = (uint32_t)f / m32;
            col = (uint32_t)f - pt * m32;
            return f < flat_total;
        } else {
            pt = t / ctiles;
            col = (t - pt * ctiles) * CSL + c;
            return col < m32;
        }
    };
    const uint32_t psh = POST == 1 ? a.tw.logN - a.post_log : 0;
    // exponent of the tile factor's part x (x = an output index): w_{2^post_log}^{+-pt x}
    auto post_exp = [&](uint32_t pt, uint32_t x) {
        uint64_t e = ((uint64_t)pt * x) << psh;
        if (INV) e = 0 - e;
        return e & mask;
    };
    // Stage 1 keeps instance row i = ((j2 / 2) S + s) 2 + (j2 & 1) in M-tile i / 128.
    auto row1_addr = [&](uint32_t i) { return Ab + (i >> 7) * (128 * 8 * R1) + (i & 127) * 16; };
    // Half `half` of the tile's inputs, HBM -> A as stage 1 reads it (two
    // halves, so that a burst of copies does not fill the memory queue; DBL
    // has only one).
    auto load = [&](uint32_t t, uint32_t half) {
        if constexpr (!DBL) {
            // R1 = 32: one row a thread, half its j1; R1 = 16: one of its two rows
            const uint32_t i = R1 == 32 ? tid : tid + half * NT, j10 = R1 == 32 ? half * 16 : 0;
            const uint32_t s = (i >> 1) % S, j2 = 2 * ((i >> 1) / S) + (i & 1);
            uint32_t pt, col;
            const bool in_range = locate(t, s, pt, col);
            const uint64_t* src =
                in_range ? a.in + ((uint64_t)pt * a.in_ts) * a.in_ld + col + (uint64_t)(j10 * R2 + j2) * ip : a.in;
            const uint64_t jstep = in_range ? R2 * ip : 0;
            const uint32_t dst = row1_addr(i) + (j10 >> 1) * 2048;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q, src += jstep)
                copy_async8(dst + (q >> 1) * 2048 + (q & 1) * 8, src, in_range);
        } else {
            // x_i, x_{i+T} -> the T-point inputs of the even and the odd outputs
            const uint32_t q = tid & 255, j10 = 16 * (tid >> 8);
            const uint32_t c = (q >> 1) & 7, j2 = 2 * (q >> 4) + (q & 1);
            uint32_t pt, col;
            const bool in_range = locate(t, c, pt, col);
            const uint64_t* src = a.in + ((uint64_t)pt * a.in_ts) * a.in_ld + col + (uint64_t)(j10 * R2 + j2) * ip;
            const uint32_t i0 = ((q >> 4) * S + c) * 2 + (q & 1);
            const uint32_t de = row1_addr(i0) + (j10 >> 1) * 2048, dodd = row1_addr(i0 + 2 * CSL) + (j10 >> 1) * 2048;
#pragma unroll
            for (uint32_t hh = 0; hh < 16; hh += 8) {
                uint64_t x[8], y[8];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    x[j] = in_range ? src[(uint64_t)((hh + j) * R2) * ip] : 0;
                    y[j] = in_range ? src[(uint64_t)((hh + j) * R2 + T) * ip] : 0;
                }
                if (gsh != 1) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) y[j] = gl::mul(y[j], gsh);
                }
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const uint64_t e = gl::add(x[j], y[j]);
                    y[j] = gl::mul(gl::sub(x[j], y[j]), W[(j10 + hh + j) * R2 + j2]);
                    x[j] = e;
                }
#pragma unroll
                for (uint32_t j = 0; j < 8; j += 2) {
                    sts128(de + ((hh + j) >> 1) * 2048, x[j], x[j + 1]);
                    sts128(dodd + ((hh + j) >> 1) * 2048, y[j], y[j + 1]);
                }
            }
        }
    };
    auto loaded = [&] {
        if constexpr (DBL) {
            fence_async();
            mbar_arrive(bar_loaded);
        } else {
            copy_async_arrive(bar_loaded);
        }
    };
    if (t0 < gtiles) {
        load(t0, 0);
        if (!DBL) load(t0, 1);
        loaded();
    }
    uint32_t odd = 0;
    for (uint32_t t = t0; t < gtiles; t += gstep, odd ^= 1) {
        uint64_t* FA = FA0 + (FLAT ? 0 : odd * PL::AB);  // a slow warp may still read the previous tile's
        uint64_t* FB = FA + A_WORDS;
        // ---- the tile's output factor w^{pt k} = a[k1] b[k2], k = D (k1 + R1 k2) + parity
        if constexpr (POST == 1) {
            if (FLAT) bar_all();
            for (uint32_t e = tid; e < PL::AB; e += NT) {
                const bool isa = e < A_WORDS;
                const uint32_t q = isa ? e : e - A_WORDS;
                const uint32_t c = FLAT ? q / (isa ? R1 : D * R2) : 0, i = FLAT ? q % (isa ? R1 : D * R2) : q;
                uint32_t pt, col;
                locate(t, c, pt, col);
                uint64_t x = isa ? post_exp(pt, D * i) : post_exp(pt, D * R1 * (i % R2) + i / R2);
                if (!isa && a.pre_kind) x += ((uint64_t)pt * a.in_ts * rep) << (a.tw.logN - a.pre_log);
                FA[e] = tw_pow(a.tw, x & mask);
            }
        }
        // all working threads are done with the previous tile; they leave together after a timeout
        if (bar_or(*abort != 0)) break;
        if constexpr (POST == 1 && !FLAT) {
            for (uint32_t e = tid; e < T; e += NT) TWX[e] = gl::mul(TW[e], FA[e / R2]);
            bar_all();
        }
        const uint64_t* TF = POST == 1 && !FLAT ? TWX : TW;
        // ---- stage 1 outputs: times the twiddles, back into A as stage 2 reads it
        stage(std::integral_constant<uint32_t, R1>{}, false,
              [&](uint32_t, uint32_t i, uint32_t k10, const uint32_t* r) {
                  const uint32_t s = (i >> 1) % S, j2 = 2 * ((i >> 1) / S) + (i & 1);
                  const uint32_t dst = Ab + (j2 >> 1) * (16 * ROWS2) + (k10 * S + s) * 16 + (j2 & 1) * 8;
                  const uint64_t* tf = TF + k10 * R2 + j2;
                  const uint64_t* fa = FA + (s % CSL) * R1 + k10;
                  uint64_t v[4];
#pragma unroll
                  for (uint32_t q = 0; q < 4; ++q) v[q] = gl::mul(recombine(r + 8 * q), tf[q * R2]);
                  if constexpr (FLAT && POST == 1) {
#pragma unroll
                      for (uint32_t q = 0; q < 4; ++q) v[q] = gl::mul(v[q], fa[q]);
                  }
#pragma unroll
                  for (uint32_t q = 0; q < 4; ++q) sts64(dst + q * S * 16, v[q]);
              });
        fence_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_ready);
        // ---- stage 2 outputs: times the output factor, to HBM
        const bool more = !DBL && t + gstep < gtiles;
        stage(std::integral_constant<uint32_t, R2>{}, true,
              [&](uint32_t step, uint32_t i, uint32_t k20, const uint32_t* r) {
                  if (more && step >= 2 && !(k20 & 4)) {
                      load(t + gstep, step - 2);
                      if (step == 3) loaded();
                  }
                  const uint32_t s = i % S, k1 = i / S, par = s / CSL, c = s % CSL;
                  uint32_t pt, col;
                  const bool in_range = locate(t, c, pt, col);
                  const uint64_t row0 = (uint64_t)pt * a.out_ts + (uint64_t)rep * a.out_rs;
                  const uint32_t k = D * (k1 + R1 * k20) + par;
                  uint64_t* dst = a.out + (row0 + (uint64_t)k * a.out_ps) * a.out_ld + col;
                  const uint64_t* fb = FB + (FLAT ? c * (D * R2) : 0) + par * R2 + k20;
                  const uint64_t ostep = (uint64_t)(D * R1) * op;
                  uint64_t f[4], v[4];
                  if constexpr (POST == 2) {
                      const uint64_t* w = a.weights + row0 + (uint64_t)k * a.out_ps;
#pragma unroll
                      for (uint32_t q = 0; q < 4; ++q) f[q] = in_range ? __ldg(w + (uint64_t)(D * R1 * q) * a.out_ps) : 0;
                  }
#pragma unroll
                  for (uint32_t q = 0; q < 4; ++q) v[q] = recombine(r + 8 * q);
#pragma unroll
                  for (uint32_t q = 0; q < 4; ++q) {
                      if constexpr (POST == 1) v[q] = gl::mul(v[q], fb[q]);
                      if constexpr (POST == 2) v[q] = gl::mul(v[q], f[q]);
                      if constexpr (POST == 3) v[q] = gl::mul(v[q], a.scalar);
                      if constexpr (POST == 0 || POST == 3) v[q] = gl::canon(v[q]);
                  }
                  if (in_range) {
#pragma unroll
                      for (uint32_t q = 0; q < 4; ++q, dst += ostep) *dst = v[q];
                  }
              });
        if (DBL && t + gstep < gtiles) {
            load(t + gstep, 0);
            loaded();
        }
    }
    // every product has been waited for above; after a timeout the issuing warp
    // waits for those in flight, and the columns are given back all the same
    copy_async_wait();
    tc_before();
    __syncthreads();
    tc_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(ctrl[0]), "n"(TMEM_COLS));
}

template <int LR1, int LR2, bool DBL, bool INV, bool FLAT, int POST>
int launch(Ctx* ctx, cudaStream_t st, const PassArgs& a, uint64_t ntiles) {
    using PL = TcPlan<LR1, LR2, DBL, FLAT>;
    KernelInfo ki;
    SG_TRY(kernel_info((const void*)k_dft_tc<LR1, LR2, DBL, INV, FLAT, POST>, PL::SMEM, NT + 32, &ki));
    const uint64_t ctiles = (a.m + PL::CSL - 1) / PL::CSL, flat = ntiles * a.m;
    const uint64_t gtiles = FLAT ? (flat + PL::CSL - 1) / PL::CSL : ntiles * ctiles;
    // log2 of the cosets the T-point DFTs are shifts of: input i of coset rep
    // carries w_{2^pre_log}^{in_ps i rep}, and 2^pre_log / in_ps = reps L
    const uint32_t lb = a.pre_kind ? a.pre_log - (uint32_t)log2_exact(a.in_ps) - LR1 - LR2 : 0;
    uint64_t per_rep = (uint64_t)ki.sms / a.reps;
    if (per_rep > gtiles) per_rep = gtiles;
    k_dft_tc<LR1, LR2, DBL, INV, FLAT, POST><<<(unsigned)(per_rep * a.reps), NT + 32, PL::SMEM, st>>>(
        a, (uint32_t)gtiles, (uint32_t)ctiles, flat, lb, ctx->fault_dev);
    return check_launch(ctx, "k_dft_tc");
}

template <int LR1, int LR2, bool DBL, bool FLAT>
int launch_kind(Ctx* ctx, cudaStream_t st, const PassArgs& a, uint64_t ntiles) {
    if (!a.inverse)
        return a.post_kind ? launch<LR1, LR2, DBL, false, FLAT, 1>(ctx, st, a, ntiles)
                           : launch<LR1, LR2, DBL, false, FLAT, 0>(ctx, st, a, ntiles);
    return a.post_kind == 1   ? launch<LR1, LR2, DBL, true, FLAT, 1>(ctx, st, a, ntiles)
           : a.post_kind == 2 ? launch<LR1, LR2, DBL, true, FLAT, 2>(ctx, st, a, ntiles)
                              : launch<LR1, LR2, DBL, true, FLAT, 3>(ctx, st, a, ntiles);
}

// Columns of a tile of 2^logL points (TcPlan::CSL).
uint64_t tile_cols(uint32_t logL) { return PTS >> logL; }

// Columns in tiles of their own leave the last one partly empty; narrow
// matrices (LogUp columns, composition parts) take their slots from the flat
// list of (tile, column) pairs instead, at one product more a point: worth it
// from an eighth of the slots (2^18 x 77, blowup 2, a fifth empty: 1.10 ms
// against 1.03 flat).
bool flat_tiles(uint64_t m, uint64_t csl) { return (m + csl - 1) / csl * csl * 8 > m * 9; }

// Whether a short pass is quicker here than on the integer pipes. All SMs take
// a tile each and the last round is as long as a full one, while k_dft's time
// grows with its points, columns padded to its narrowest tile; so a pass of
// 70 or of 150 tiles may be the slower one here. Both times in tenths of a
// microsecond, fitted to 944 passes of LDEs of 2^7..2^22 rows x 1..600
// columns, blowup 1 to 16: the quicker kernel is taken but for eight passes
// that lose 3 to 20 %. 2^14 x 77, blowup 2: 116 us with every pass over 2^20
// points here, 91 without any. Passes of 2^10 and 2^11 points are quicker here
// at every size measured (1.14 to 5 times), and so are those over more than
// two cosets, which k_dft runs one after another in a tile (up to 5 times).
bool quicker_here(const PassArgs& a, uint64_t ntiles) {
    if (a.logL > 9 || a.reps > 2) return true;
    struct Times {
        uint64_t round, lead, mpoint;  // a round here; what k_dft starts later, its time for 2^20 points
    };
    static constexpr Times T[3] = {{140, 10, 85}, {146, 50, 91}, {164, 30, 107}};  // 2^7, 2^8, 2^9 points
    const Times& t = T[a.logL - 7];
    const uint64_t csl = tile_cols(a.logL), narrowest = a.logL == 7 ? 32 : 4, ctas = 148 / a.reps;
    const bool flat = flat_tiles(a.m, csl);
    const uint64_t tiles = flat ? (ntiles * a.m + csl - 1) / csl : ntiles * ((a.m + csl - 1) / csl);
    const uint64_t rounds = (tiles + ctas - 1) / ctas;
    const uint64_t padded = ((a.m + narrowest - 1) / narrowest * narrowest * ntiles * a.reps) << a.logL;
    const uint64_t more = (flat ? 8 : 0) + (a.inverse ? 15 : a.post_kind == 1 ? 10 : 0);
    return rounds * (t.round + more) <= t.lead + (t.mpoint * padded >> 20);
}

template <int LR1, int LR2, bool DBL>
int launch_len(Ctx* ctx, cudaStream_t st, const PassArgs& a, uint64_t ntiles) {
    static_assert(TcPlan<LR1, LR2, DBL, false>::CSL == PTS >> (LR1 + LR2 + DBL), "columns of a tile");
    return flat_tiles(a.m, tile_cols(a.logL)) ? launch_kind<LR1, LR2, DBL, true>(ctx, st, a, ntiles)
                                              : launch_kind<LR1, LR2, DBL, false>(ctx, st, a, ntiles);
}

}  // namespace

bool dft_tc_takes(const PassArgs& a, uint64_t ntiles) {
    if (a.logL < 7 || a.logL > 11) return false;
    // the kinds of the LDE's and the transforms' passes: forward with the
    // four-step factor or canonical output, inverse with either factor or 1/n
    const bool canon = a.post_kind == 0 || a.post_kind == 3;
    if ((a.canon_out != 0) != canon || (a.inverse ? a.post_kind == 0 : a.post_kind > 1)) return false;
    const uint64_t L = 1ull << a.logL;
    // the tile's part of the coset shift rides on the four-step factor
    if (a.pre_kind && (a.inverse || (a.post_kind != 1 && ntiles != 1) || log2_exact(a.in_ps) < 0)) return false;
    if (a.reps > 1 && !a.pre_kind) return false;
    if (a.reps < 1 || a.reps > 16 || log2_exact(a.reps) < 0) return false;
    // 32-bit tile and column arithmetic
    if (a.m >= (1ull << 24) || ntiles * a.m >= (1ull << 31)) return false;
    // Set-up (matrices, twiddles, TMEM) costs a CTA about 8 us and a tile takes
    // another 8: up to 64 tiles the integer kernel's many small CTAs are quicker.
    return L * ntiles * a.m * a.reps > TC_MIN_POINTS && quicker_here(a, ntiles);
}

int launch_dft_tc(Ctx* ctx, cudaStream_t st, const PassArgs& a, uint64_t ntiles) {
    switch (a.logL) {
        case 7: return launch_len<4, 3, false>(ctx, st, a, ntiles);
        case 8: return launch_len<4, 4, false>(ctx, st, a, ntiles);
        case 9: return launch_len<4, 5, false>(ctx, st, a, ntiles);
        case 10: return launch_len<5, 5, false>(ctx, st, a, ntiles);
        case 11: return launch_len<5, 5, true>(ctx, st, a, ntiles);
        default: set_error("no tensor-core DFT of this length"); return SG_ERR_UNSUPPORTED;
    }
}

}  // namespace sg
