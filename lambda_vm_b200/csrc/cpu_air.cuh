// The RV64 CPU and SHIFT tables' layouts, and their constraints as
// hand-written kernels.
//
// The CPU table (lambda_vm_b200/rv64_air.py CpuAir) has 200 or 234 columns
// and ~300 base-field constraints (one-hot selectors, operand reads from the
// register file carried in the row, 32-bit limb arithmetic, the register-file
// transitions). This kernel evaluates them directly, eight warps to 32 LDE
// rows, and folds them into the composition with the CpuAir emission order's
// constraint indices, so its sum equals the constraint walk's exactly. The
// chips the proof carries (bitwise, shift, memory, keccak) decide which
// constraint blocks exist, as in CpuAir. The LogUp constraints come from the
// table's descriptor (k_logup_constraints).
#pragma once

#include <stdint.h>

#include "gl.cuh"
#include "keccak_air.cuh"
#include "tc.cuh"

namespace sg {

// Column layout of the CPU table: the core columns and the register file
// (CPU_CORE_WIDTH), then the chips' columns. Selector of op id i (1-based,
// rv64.py OPS order, 18 = the keccak ecall): CPU_SEL0 + i - 1.
constexpr uint32_t CPU_PC = 0, CPU_STEP = 1, CPU_CLK = 2, CPU_SEL0 = 3, CPU_RD0 = 21, CPU_RS10 = 53, CPU_RS20 = 85,
                   CPU_IMM_LO = 117, CPU_IMM_HI = 118, CPU_IMM_F = 119, CPU_A_LO = 120, CPU_A_HI = 121,
                   CPU_B_LO = 122, CPU_B_HI = 123, CPU_R_LO = 124, CPU_R_HI = 125, CPU_R16 = 126, CPU_C0 = 130,
                   CPU_C1 = 131, CPU_INV_LO = 132, CPU_INV_HI = 133, CPU_E_LO = 134, CPU_E_HI = 135, CPU_NE = 136,
                   CPU_BR = 137, CPU_X0 = 138, CPU_CORE_WIDTH = 200, CPU_AB0 = 200, CPU_BB0 = 208, CPU_RB0 = 216,
                   CPU_MA = 224, CPU_MW0 = 225, CPU_MW1 = 226, CPU_MV_LO = 227, CPU_MV_HI = 228, CPU_MT = 229,
                   CPU_MD0 = 230, CPU_MD1 = 231, CPU_NV_LO = 232, CPU_NV_HI = 233, CPU_FULL_WIDTH = 234;
enum CpuOp : uint32_t {
    OPC_ADD = 1, OPC_SUB, OPC_ADDI, OPC_LUI, OPC_BEQ, OPC_BNE, OPC_ECALL, OPC_XOR, OPC_OR, OPC_AND, OPC_XORI,
    OPC_ORI, OPC_ANDI, OPC_SLLI, OPC_SRLI, OPC_LD, OPC_SD, OPC_KECCAK
};
constexpr uint32_t CHIP_BITWISE = 1, CHIP_SHIFT = 2, CHIP_MEMORY = 4, CHIP_KECCAK = 8;

// The number of base constraints CpuAir emits for a chip set.
__host__ __device__ constexpr uint32_t cpu_air_constraints(uint32_t chips) {
    const bool bw = chips & CHIP_BITWISE, sh = chips & CHIP_SHIFT, mem = chips & CHIP_MEMORY,
               kc = chips & CHIP_KECCAK;
    const uint32_t absent = (bw ? 0 : 6) + (sh ? 0 : 2) + (mem ? 0 : 2) + ((kc && mem) ? 0 : 1);
    return 117 + 4 + absent + 30 + (bw ? 6 : 0) + (mem ? 12 : 0) + 64 + 65;
}

// A SHIFT-table row, from the column-major copy (cm) or the LDE (rm).
struct CRow {
    const uint64_t* cm;
    const uint64_t* rm;
    uint64_t rows, width, row;
    __device__ __forceinline__ uint64_t M(uint32_t col) const {
        return cm ? cm[(uint64_t)col * rows + row] : rm[row * width + col];
    }
};

__device__ __forceinline__ uint32_t cpu_xlo(uint32_t k) { return CPU_X0 + 2 * (k - 1); }

// Rows of a tile, and the warps that share them: lane = row, and every warp
// evaluates its own part of the constraints of all 32 rows. The tile is copied
// from the row-major LDE in whole row segments, all copies in flight together,
// and kept column-major in shared memory (pitch 33: no bank conflicts). One
// thread a row, reading its row's columns straight from the LDE, touched 32
// rows' sectors per load and waited for them. 2^20 rows: 3.0 ms that way, 3.1
// with a tile loaded through registers (row by row, each waiting for the
// last), 2.5 here; two tiles an SM, 39 % of the issue slots used, the rest
// waits on the copies and at the tile's barriers.
constexpr uint32_t CPU_TILE = 32, CPU_WARPS = 8, CPU_PITCH = CPU_TILE + 1;
// The columns read of the next frame row: pc, timestamp, the register file.
constexpr uint32_t CPU_NEXT = 2 + 62;
__host__ __device__ constexpr size_t cpu_air_smem(uint32_t width) {
    return ((size_t)(width + CPU_NEXT) * CPU_PITCH + CPU_WARPS * CPU_TILE * 3) * 8;
}

struct CpuTile {
    const uint64_t* m;  // columns of this row, CPU_PITCH apart
    const uint64_t* n;  // the CPU_NEXT columns of the next frame row
    __device__ __forceinline__ uint64_t M(uint32_t col) const { return m[col * CPU_PITCH]; }
    __device__ __forceinline__ uint64_t sel(uint32_t op) const { return M(CPU_SEL0 + op - 1); }
    __device__ __forceinline__ uint64_t N_pc() const { return n[0]; }
    __device__ __forceinline__ uint64_t N_clk() const { return n[CPU_PITCH]; }
    // register k's limb
    __device__ __forceinline__ uint64_t x(uint32_t k, uint32_t limb) const { return M(cpu_xlo(k) + limb); }
    __device__ __forceinline__ uint64_t N_x(uint32_t k, uint32_t limb) const {
        return n[(2 + 2 * (k - 1) + limb) * CPU_PITCH];
    }
};

static __global__ void __launch_bounds__(CPU_WARPS * 32, 2)
    k_cpu_constraints(const uint64_t* __restrict__ rm, uint32_t width, uint64_t rows, uint64_t next_step,
                      uint32_t chips, const uint64_t* __restrict__ beta, int mode, uint64_t* __restrict__ out) {
    extern __shared__ uint64_t cpu_sm[];
    uint64_t* tm = cpu_sm;
    uint64_t* tn = tm + width * CPU_PITCH;
    uint64_t* part = tn + CPU_NEXT * CPU_PITCH;
    const uint64_t K32 = 1ull << 32, K16 = 1ull << 16;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // indices of the constraint blocks in CpuAir's order
    const bool bw = chips & CHIP_BITWISE, sh = chips & CHIP_SHIFT, mem = chips & CHIP_MEMORY,
               kc = (chips & CHIP_KECCAK) && mem;
    const uint32_t c_absent = 121, c_read = c_absent + (bw ? 0 : 6) + (sh ? 0 : 2) + (mem ? 0 : 2) + (kc ? 0 : 1),
                   c_arith = c_read + 4, c_bw = c_arith + 26, c_mem = c_bw + (bw ? 6 : 0),
                   c_trans = c_mem + (mem ? 12 : 0), c_end = c_trans + 64;
    for (uint64_t r0 = (uint64_t)blockIdx.x * CPU_TILE; r0 < rows; r0 += (uint64_t)gridDim.x * CPU_TILE) {
        __syncthreads();  // the previous tile is done with
        for (uint32_t r = warp; r < CPU_TILE; r += CPU_WARPS) {
            const uint64_t row = r0 + r < rows ? r0 + r : rows - 1;
            const uint64_t rn = row + next_step >= rows ? row + next_step - rows : row + next_step;
            const uint64_t *p = rm + row * width, *q = rm + rn * width;
            const uint32_t to = tc::smem_addr(tm + r), tq = tc::smem_addr(tn + r);
            for (uint32_t c = lane; c < width; c += 32) tc::copy_async8(to + c * (CPU_PITCH * 8), p + c, true);
            for (uint32_t c = lane; c < CPU_NEXT; c += 32)
                tc::copy_async8(tq + c * (CPU_PITCH * 8), q + (c == 0 ? CPU_PC : c == 1 ? CPU_CLK : CPU_X0 + c - 2), true);
        }
        tc::copy_async_wait();
        __syncthreads();
        // lanes past the end have the last row's cells and, per constraint, write its values again
        const uint64_t row = r0 + lane < rows ? r0 + lane : rows - 1;
        const CpuTile w{tm + lane, tn + lane};
        KSink s{beta, mode, out, rows, row, gl::wzero3(), 0};
        const uint64_t step = w.M(CPU_STEP), c0 = w.M(CPU_C0), c1 = w.M(CPU_C1);
        const uint64_t rl = w.M(CPU_R_LO), rh = w.M(CPU_R_HI), al = w.M(CPU_A_LO), ah = w.M(CPU_A_HI),
                       bl = w.M(CPU_B_LO), bh = w.M(CPU_B_HI), il = w.M(CPU_IMM_LO), ih = w.M(CPU_IMM_HI);
        const uint64_t s_ecall = w.sel(OPC_ECALL), s_kec = w.sel(OPC_KECCAK), s_ld = w.sel(OPC_LD), s_sd = w.sel(OPC_SD);
        // ---- every warp: a share of the booleans
        for (uint32_t i = warp; i < 18; i += CPU_WARPS) s.put(3 + i, kbool(w.M(CPU_SEL0 + i)));
        for (uint32_t i = warp; i < 96; i += CPU_WARPS) s.put(21 + i, kbool(w.M(CPU_RD0 + i)));
        // ---- warps 0..3: operand reads a = x[rs1], b = x[rs2], a limb each
        if (warp < 4) {
            const uint32_t op2 = warp >> 1, limb = warp & 1, base = op2 ? CPU_RS20 : CPU_RS10;
            gl::wacc t = gl::wzero();  // the 31 products summed unreduced
            for (uint32_t k = 1; k < 32; ++k) gl::wmac(t, w.M(base + k), w.x(k, limb));
            s.put(c_read + warp, gl::sub(w.M((op2 ? CPU_B_LO : CPU_A_LO) + limb), gl::wreduce(t)));
        } else {
            // ---- warps 4..7: one-hot sums (the selectors, rd, rs1, rs2)
            const uint32_t first = warp == 4 ? CPU_SEL0 : CPU_RD0 + 32 * (warp - 5), count = warp == 4 ? 18 : 32;
            uint64_t t = 0;
            for (uint32_t k = 0; k < count; ++k) t = gl::add(t, w.M(first + k));
            s.put(117 + warp - 4, gl::sub(t, 1));
        }
        // ---- warps 0..6: transitions of the register file and the END row's
        // initial state, register by register (warp 6 has the chips' blocks too)
        {
            const uint64_t nstep = gl::sub(1, step);
            const uint32_t k_lo = warp < 6 ? 1 + 5 * warp : (warp == 6 ? 31 : 32), k_hi = warp < 6 ? k_lo + 5 : 32;
            for (uint32_t k = k_lo; k < k_hi; ++k) {
                const uint64_t rdk = w.M(CPU_RD0 + k);
                for (uint32_t limb = 0; limb < 2; ++limb) {
                    const uint64_t x = w.x(k, limb), nx = w.N_x(k, limb);
                    const uint64_t upd = gl::mul(rdk, gl::sub(limb ? rh : rl, x));
                    s.put(c_trans + 2 + 2 * (k - 1) + limb, gl::mul(step, gl::sub(nx, gl::add(x, upd))));
                    s.put(c_end + 3 + 2 * (k - 1) + limb, gl::mul(nstep, nx));
                }
            }
        }
        if (warp == 6) {
            const uint64_t c0k = gl::mul(c0, K32), c1k = gl::mul(c1, K32);
            // an instruction whose chip the proof does not carry cannot occur
            uint32_t c = c_absent;
            if (!bw)
                for (uint32_t op = OPC_XOR; op <= OPC_ANDI; ++op) s.put(c++, w.sel(op));
            if (!sh) s.put(c, w.sel(OPC_SLLI)), s.put(c + 1, w.sel(OPC_SRLI)), c += 2;
            if (!mem) s.put(c, s_ld), s.put(c + 1, s_sd), c += 2;
            if (!kc) s.put(c, s_kec);
            if (bw) {
                s.next = c_bw;
                const uint64_t sreg = gl::add(gl::add(w.sel(OPC_XOR), w.sel(OPC_OR)), w.sel(OPC_AND));
                const uint64_t simm = gl::add(gl::add(w.sel(OPC_XORI), w.sel(OPC_ORI)), w.sel(OPC_ANDI));
                const uint64_t sbit = gl::add(sreg, simm);
                for (uint32_t limb = 0; limb < 2; ++limb) {
                    auto bytes = [&](uint32_t first) {
                        uint64_t t = 0;
                        for (uint32_t i = 0; i < 4; ++i)
                            t = gl::add(t, gl::mul(1ull << (8 * i), w.M(first + i + 4 * limb)));
                        return t;
                    };
                    const uint64_t a_ = limb ? ah : al, b_ = limb ? bh : bl, i_ = limb ? ih : il, r_ = limb ? rh : rl;
                    s.put(gl::mul(sbit, gl::sub(a_, bytes(CPU_AB0))));
                    const uint64_t ob = bytes(CPU_BB0);
                    s.put(gl::add(gl::mul(sreg, gl::sub(b_, ob)), gl::mul(simm, gl::sub(i_, ob))));
                    s.put(gl::mul(sbit, gl::sub(r_, bytes(CPU_RB0))));
                }
            }
            if (mem) {
                s.next = c_mem;
                const uint64_t sm = gl::add(s_ld, s_sd), saddr = gl::add(sm, s_kec), ma = w.M(CPU_MA);
                s.put(gl::mul(sm, gl::sub(gl::add(ma, c0k), gl::add(al, il))));
                s.put(gl::mul(sm, gl::sub(c1k, gl::add(gl::add(ah, ih), c0))));
                s.put(gl::mul(s_kec, gl::sub(ma, w.x(10, 0))));
                s.put(gl::mul(s_kec, w.x(10, 1)));
                s.put(gl::mul(saddr,
                              gl::sub(ma, gl::add(gl::mul(8, w.M(CPU_MW0)), gl::mul(1ull << 19, w.M(CPU_MW1))))));
                const uint64_t gap = gl::sub(gl::sub(w.M(CPU_CLK), w.M(CPU_MT)), 1);
                s.put(gl::mul(sm, gl::sub(gap, gl::add(w.M(CPU_MD0), gl::mul(K16, w.M(CPU_MD1))))));
                for (uint32_t limb = 0; limb < 2; ++limb) {
                    const uint64_t nv = w.M(limb ? CPU_NV_HI : CPU_NV_LO), mv = w.M(limb ? CPU_MV_HI : CPU_MV_LO);
                    s.put(gl::mul(s_ld, gl::sub(nv, mv)));
                    s.put(gl::mul(s_sd, gl::sub(nv, limb ? bh : bl)));
                    s.put(gl::mul(s_ld, gl::sub(limb ? rh : rl, mv)));
                }
            }
        }
        if (warp == 7) {
            s.put(0, kbool(step));
            s.put(1, kbool(c0));
            s.put(2, kbool(c1));
            s.next = c_arith;
            // the written value in 16-bit pieces
            s.put(gl::sub(rl, gl::add(w.M(CPU_R16), gl::mul(K16, w.M(CPU_R16 + 1)))));
            s.put(gl::sub(rh, gl::add(w.M(CPU_R16 + 2), gl::mul(K16, w.M(CPU_R16 + 3)))));
            // add / addi, sub, lui
            const uint64_t s_add = w.sel(OPC_ADD), s_addi = w.sel(OPC_ADDI), s_sub = w.sel(OPC_SUB),
                           s_lui = w.sel(OPC_LUI);
            const uint64_t c0k = gl::mul(c0, K32), c1k = gl::mul(c1, K32);
            s.put(gl::mul(s_add, gl::sub(gl::add(rl, c0k), gl::add(al, bl))));
            s.put(gl::mul(s_add, gl::sub(gl::add(rh, c1k), gl::add(gl::add(ah, bh), c0))));
            s.put(gl::mul(s_addi, gl::sub(gl::add(rl, c0k), gl::add(al, il))));
            s.put(gl::mul(s_addi, gl::sub(gl::add(rh, c1k), gl::add(gl::add(ah, ih), c0))));
            s.put(gl::mul(s_sub, gl::sub(gl::add(rl, bl), gl::add(al, c0k))));
            s.put(gl::mul(s_sub, gl::sub(gl::add(gl::add(rh, bh), c0), gl::add(ah, c1k))));
            s.put(gl::mul(s_lui, gl::sub(rl, il)));
            s.put(gl::mul(s_lui, gl::sub(rh, ih)));
            // no value for branches, ecalls and stores; carries only where an addition uses them
            const uint64_t s_beq = w.sel(OPC_BEQ), s_bne = w.sel(OPC_BNE);
            const uint64_t nores = gl::add(gl::add(gl::add(gl::add(s_beq, s_bne), s_ecall), s_kec), s_sd);
            s.put(gl::mul(nores, rl));
            s.put(gl::mul(nores, rh));
            const uint64_t nocarry = gl::sub(1, gl::add(gl::add(gl::add(gl::add(s_add, s_addi), s_sub), s_ld), s_sd));
            s.put(gl::mul(nocarry, c0));
            s.put(gl::mul(nocarry, c1));
            // branch witnesses
            const uint64_t branch = gl::add(s_beq, s_bne);
            const uint64_t el = w.M(CPU_E_LO), eh = w.M(CPU_E_HI);
            for (uint32_t limb = 0; limb < 2; ++limb) {
                const uint64_t d = limb ? gl::sub(ah, bh) : gl::sub(al, bl);
                const uint64_t e = limb ? eh : el, inv = w.M(limb ? CPU_INV_HI : CPU_INV_LO);
                s.put(gl::mul(branch, gl::sub(e, gl::mul(d, inv))));
                s.put(gl::mul(branch, gl::mul(d, gl::sub(1, e))));
                s.put(gl::mul(gl::sub(1, branch), e));
            }
            const uint64_t ne = w.M(CPU_NE), br = w.M(CPU_BR);
            s.put(gl::sub(ne, gl::sub(gl::add(el, eh), gl::mul(el, eh))));
            s.put(gl::sub(br, gl::add(gl::mul(s_beq, gl::sub(1, ne)), gl::mul(s_bne, ne))));
            // ecalls: exit with a7 = 93, keccak with a7 = 2^64 - 2
            const uint64_t x17l = w.x(17, 0), x17h = w.x(17, 1);
            s.put(gl::mul(s_ecall, gl::sub(x17l, 93)));
            s.put(gl::mul(s_ecall, x17h));
            s.put(gl::mul(s_kec, gl::sub(x17l, 0xFFFFFFFEull)));
            s.put(gl::mul(s_kec, gl::sub(x17h, 0xFFFFFFFFull)));
            // transitions: next pc, timestamp
            const uint64_t adv = gl::add(gl::mul(4, gl::sub(1, s_ecall)), gl::mul(br, gl::sub(w.M(CPU_IMM_F), 4)));
            s.put(c_trans, gl::mul(step, gl::sub(w.N_pc(), gl::add(w.M(CPU_PC), adv))));
            s.put(c_trans + 1, gl::mul(step, gl::sub(w.N_clk(), gl::add(w.M(CPU_CLK), 1))));
            // the END row: an exit ecall, followed by the initial state
            const uint64_t nstep = gl::sub(1, step);
            s.put(c_end, gl::mul(nstep, gl::sub(1, s_ecall)));
            s.put(c_end + 1, gl::mul(nstep, w.N_pc()));
            s.put(c_end + 2, gl::mul(nstep, gl::sub(w.N_clk(), 1)));
        }
        if (mode == 0) {
            const gl::fe3 sum = s.total();
            uint64_t* o = part + 3 * threadIdx.x;
            o[0] = sum.c0, o[1] = sum.c1, o[2] = sum.c2;
            __syncthreads();
            // one thread a (row, component): the warps' sums together
            if (threadIdx.x < 3 * CPU_TILE) {
                const uint32_t r = threadIdx.x / 3, k = threadIdx.x % 3;
                uint64_t t = part[3 * r + k];
                for (uint32_t v = 1; v < CPU_WARPS; ++v) t = gl::add(t, part[3 * (32 * v + r) + k]);
                if (r0 + r < rows) out[3 * (r0 + r) + k] = t;
            }
        }
    }
}

// The SHIFT table (rv64_air.py ShiftAir): DIR, the operand's bits, one-hot
// s = k mod 8 and q = k div 8, the operand shifted by s bits, the result's
// limbs, the multiplicity. Its 149 base constraints in ShiftAir's order.
constexpr uint32_t SH_DIR = 0, SH_AB = 1, SH_S = 65, SH_Q = 73, SH_TB = 81, SH_R_LO = 145, SH_R_HI = 146,
                   SH_WIDTH = 148, SH_CONSTRAINTS = 149;

static __global__ void k_shift_constraints(const uint64_t* __restrict__ cm, const uint64_t* __restrict__ rm,
                                           uint64_t rows, const uint64_t* __restrict__ beta, int mode,
                                           uint64_t* __restrict__ out) {
    for (uint64_t row = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
         row += (uint64_t)gridDim.x * blockDim.x) {
        const CRow w{cm, rm, rows, SH_WIDTH, row};
        KSink s{beta, mode, out, rows, row, gl::wzero3(), 0};
        const uint64_t d = w.M(SH_DIR), nd = gl::sub(1, d);
        s.put(kbool(d));
        for (uint32_t i = 0; i < 64; ++i) s.put(kbool(w.M(SH_AB + i)));
        for (uint32_t i = 0; i < 8; ++i) s.put(kbool(w.M(SH_S + i)));
        for (uint32_t i = 0; i < 8; ++i) s.put(kbool(w.M(SH_Q + i)));
        uint64_t ts = 0, tq = 0;
        for (uint32_t i = 0; i < 8; ++i) ts = gl::add(ts, w.M(SH_S + i)), tq = gl::add(tq, w.M(SH_Q + i));
        s.put(gl::sub(ts, 1));
        s.put(gl::sub(tq, 1));
        // TB_j = sum_s S_s (nd a[j - s] + d a[j + s]), bits past either end
        // zero, evaluated as nd (sum_s S_s a[j - s]) + d (sum_s S_s a[j + s])
        // with both sums kept unreduced (the same polynomial)
        uint64_t sv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) sv[k] = w.M(SH_S + k);
        // four bits at a time, their 18 operand bits read once into registers
        // (16 reads a bit, two per product, were what bound this kernel)
        for (int j0 = 0; j0 < 64; j0 += 4) {
            uint64_t ab[18];  // a[j0 - 7 .. j0 + 10]
#pragma unroll
            for (int i = 0; i < 18; ++i) ab[i] = (unsigned)(j0 + i - 7) < 64u ? w.M(SH_AB + j0 + i - 7) : 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                gl::wacc lo = gl::wzero(), hi = gl::wzero();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    gl::wmac(lo, sv[k], ab[7 + i - k]);
                    gl::wmac(hi, sv[k], ab[7 + i + k]);
                }
                const uint64_t t = gl::add(gl::mul(nd, gl::wreduce(lo)), gl::mul(d, gl::wreduce(hi)));
                s.put(gl::sub(w.M(SH_TB + j0 + i), t));
            }
        }
        // the result moves TB by whole bytes: byte k = sum_q Q_q (nd tB[k - q] + d tB[k + q])
        uint64_t tB[8];
        for (int i = 0; i < 8; ++i) {
            uint64_t t = 0;
            for (int j = 7; j >= 0; --j) t = gl::add(gl::add(t, t), w.M(SH_TB + 8 * i + j));
            tB[i] = t;
        }
        uint64_t qv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) qv[q] = w.M(SH_Q + q);
        for (int limb = 0; limb < 2; ++limb) {
            uint64_t acc = 0;
            for (int k = 4 * limb + 3; k >= 4 * limb; --k) {
                gl::wacc lo = gl::wzero(), hi = gl::wzero();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (k - q >= 0) gl::wmac(lo, qv[q], tB[k - q]);
                    if (k + q < 8) gl::wmac(hi, qv[q], tB[k + q]);
                }
                const uint64_t t = gl::add(gl::mul(nd, gl::wreduce(lo)), gl::mul(d, gl::wreduce(hi)));
                acc = gl::add(gl::mul(acc, 256), t);
            }
            s.put(gl::sub(w.M(limb ? SH_R_HI : SH_R_LO), acc));
        }
        if (mode == 0) {
            uint64_t* o = out + 3 * row;
            const gl::fe3 sum = s.total();
            o[0] = sum.c0, o[1] = sum.c1, o[2] = sum.c2;
        }
    }
}

}  // namespace sg
