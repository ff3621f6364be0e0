// FP32 SIMT GEMM for sm_100a: C = A*B, row-major, on the CUDA cores.
//
// Replaces the reference's blocked SME driver (sme/v3/sme-1x4-acc-kcout.cpp:427-567)
// as the FP32-accurate path. The SME packers (pack_A_streaming :39-136,
// pack_B_streaming :145-193) become a ring of shared-memory stages filled by
// cp.async; the 16x64 ZA micro-tile becomes a CTA tile of tile_m x tile_n with
// a register tile of packed FP32 pairs per thread.
//
// Arithmetic: every output is ONE sequential chain over k in increasing order
// (a fused multiply-add per step, or multiply-then-add in the SCALAR variant,
// the arithmetic of Utils::multiply_scalar, common/utils.hpp:50-61). With
// split_k > 1 each K slice is such a chain and the slices are summed in slice
// order, first slice first: C = ((p0 + p1) + p2) + ..., the order in which
// the reference's v3 adds its outer-Kc panels (first_k store, then
// store_za_add; sme/v3/sme-1x4-acc-kcout.cpp:464-471, 530-558). The result is
// therefore deterministic and reproducible bit for bit by a scalar loop.
//
// Edges (the reference's scratch-tile path, :539-558) are predicated loads
// that read zero outside the matrix and predicated stores; C outside the
// matrix is never touched.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

#include "internal.hpp"
#include "launch.cuh"
#include "phase.hpp"
#include "runtime.hpp"
#include "split_math.cuh"

namespace mmsk {
namespace {

// The end of one tile: without a K split the sums go to C; with one, this
// slice's partial tile is written and, unless a separate reduction kernel
// follows, the last CTA of the tile to arrive sums all slices in slice order
// (C = ((p0 + p1) + p2) + ...). acc[i][4 g + j] is the output at row
// out_row(i), column out_col(g) + j. `last_flag` is a shared-memory word.
template <int TM, int GN, class RowFn, class ColFn>
__device__ __forceinline__ void simt_epilogue(const SimtArgs& p, float (&acc)[TM][4 * GN], RowFn out_row,
                                              ColFn out_col, bool VEC, int z, unsigned tile, int& last_flag) {
    const int64_t M = p.M, N = p.N;
    const int tid = threadIdx.x;
    if (p.splits <= 1) {
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const int64_t r = out_row(i);
            if (r >= M) continue;
#pragma unroll
            for (int g = 0; g < GN; g++) {
                const int64_t c = out_col(g);
                float* dst = p.C + r * N + c;
                if (VEC && c + 3 < N) {
                    *reinterpret_cast<float4*>(dst) =
                        make_float4(acc[i][g * 4 + 0], acc[i][g * 4 + 1], acc[i][g * 4 + 2], acc[i][g * 4 + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (c + j < N) dst[j] = acc[i][g * 4 + j];
                }
            }
        }
        return;
    }

    // Split-K: write this slice's partial tile, then the last CTA of the tile
    // to arrive sums all slices in slice order.
    const size_t MN = (size_t)M * (size_t)N;
    float* mine = p.partial + (size_t)z * MN;
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int64_t r = out_row(i);
        if (r >= M) continue;
#pragma unroll
        for (int g = 0; g < GN; g++) {
            const int64_t c = out_col(g);
            if (VEC && c + 3 < N) {
                __stcg(reinterpret_cast<float4*>(mine + r * N + c),
                       make_float4(acc[i][g * 4 + 0], acc[i][g * 4 + 1], acc[i][g * 4 + 2], acc[i][g * 4 + 3]));
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (c + j < N) __stcg(mine + r * N + c + j, acc[i][g * 4 + j]);
            }
        }
    }
    if (p.reduce_after) return;                      // summed by simt_splitk_reduce_kernel
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned prev = atomicAdd(&p.counters[tile], 1u);
        last_flag = (prev == (unsigned)(p.splits - 1));
    }
    __syncthreads();
    const int last = last_flag;
    __syncthreads();                                 // the flag may be rewritten by the next tile
    if (!last) return;
    __threadfence();
    // Each output: slice 0, then every later slice added in slice order; four
    // adjacent columns at a time with 128-bit loads where rows allow.
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int64_t r = out_row(i);
        if (r >= M) continue;
#pragma unroll
        for (int g = 0; g < GN; g++) {
            const int64_t c = out_col(g);
            const size_t off = (size_t)r * N + c;
            if (VEC && c + 3 < N) {
                float4 s4 = __ldcg(reinterpret_cast<const float4*>(p.partial + off));
                for (int q = 1; q < p.splits; q++) {
                    const float4 t = __ldcg(reinterpret_cast<const float4*>(p.partial + (size_t)q * MN + off));
                    s4.x = __fadd_rn(s4.x, t.x); s4.y = __fadd_rn(s4.y, t.y);
                    s4.z = __fadd_rn(s4.z, t.z); s4.w = __fadd_rn(s4.w, t.w);
                }
                *reinterpret_cast<float4*>(p.C + off) = s4;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (c + j >= N) continue;
                    float v = __ldcg(p.partial + off + j);
                    for (int q = 1; q < p.splits; q++) v = __fadd_rn(v, __ldcg(p.partial + (size_t)q * MN + off + j));
                    p.C[off + j] = v;
                }
            }
        }
    }
    if (tid == 0) p.counters[tile] = 0u;   // leave the counter ready for the next call
}

// ---------------------------------------------------------------------------
// The tile kernel: packed multiply-adds on a cp.async ring.
//
// A warp owns 8 RT x 4 LT outputs; lane = 4 lm + ln holds rows lm + 8 i (i <
// RT) and columns 4 ln + 16 j + {0..3} (j < LT / 4) of them as RT x LT / 2
// packed pairs. Stages of BK k's of A (rows padded to BK + 4 floats, so a
// warp's eight rows fall on eight bank groups) and B arrive by cp.async in the
// widest copies the operand's alignment allows (SimtArgs::wa, wb).
//
// Bound by the FMA pipe: 128 multiply-adds per clock and SM, 74.4 TFLOP/s at
// 1965 MHz. fma.rn.f32x2 issues half as many instructions for the same pipe
// cycles, which leaves issue slots for the shared loads; operands are
// duplicated into pairs from A, RT moves per RT LT / 2 instructions. Register
// operand conflicts hold a loop of nothing but these instructions to 88-91 %
// of the peak by the order they come in. Measured at 4096^3, 128 x 128 tiles,
// no K split: 2358 us (58.3 TFLOP/s) against 3011 us with scalar multiply-adds
// and fragments read from shared memory where they are used; 2620 us with
// packed ones alone, 2477 us with fragments read one k ahead across stage
// boundaries, 2397 us with the column-snake order below (row by row 2477,
// row snake 2459, 2 x 2 blocks 2479), 2358 us with bounds tested per stage
// rather than per copy. A sizes of K and N that are not multiples of 4 cost 12 %
// over their aligned neighbours (776 x 1531 x 899 and 776 x 1532 x 900: 75.2
// and 67.4 us; 108.6 and 101.7 us before, 94.7 us with bounds per copy).
//
// Arithmetic: every output is one chain over k in increasing order, so C is
// the same bit for bit whatever the tile; copies past kend write zeros.
// ---------------------------------------------------------------------------
template <int BM_, int BN_, int RT_, int LT_, int BK_, int STAGES_, int CTAS_, int LM_ = 8>
struct CpCfg {
    static constexpr int BM = BM_, BN = BN_, RT = RT_, LT = LT_, BK = BK_, STAGES = STAGES_, CTAS = CTAS_;
    static constexpr int LM = LM_, LN = 32 / LM;    // lanes along M and N
    static constexpr int WM = LM * RT, WN = LN * LT;  // warp tile
    static constexpr int WARPS_N = BN / WN;
    static constexpr int THREADS = 32 * (BM / WM) * WARPS_N;
    static constexpr int AST = BK + 4;             // A row stride (floats): eight rows on eight bank groups
    static constexpr int A_FLOATS = BM * AST;
    static constexpr int B_FLOATS = BK * BN;
    static constexpr int STAGE_FLOATS = A_FLOATS + B_FLOATS;
    static constexpr int SMEM = STAGES * STAGE_FLOATS * 4;
    static_assert(THREADS >= BK && BK % 4 == 0 && STAGES >= 3 && THREADS <= 4 * BN, "tile configuration");
};

// The plans' tiles. 128 x 128: 8 x 16 outputs a thread (244 registers; 255 and 8
// bytes spilled in the SCALAR variant; two CTAs an SM). 128 x 64: 8 x 8 a thread. 64 x 64: 4 x 8 a thread and four CTAs
// an SM, which a small C needs to fill the GPU. Measured, per configuration
// (4096^3 unsplit, 128 x 128: BK 16 x 4 stages 2358 us, 16 x 3 2377, 8 x 6
// 2496; 2048^3 split 2, 128 x 64: 32 x 3, two CTAs 344, 16 x 4, three CTAs
// 350; 2048^3 unsplit, 64 x 64: 32 x 3 354, 16 x 4 394, 4 x 4 a thread 475).
template <int BM, int BN> struct CpTileSel;
template <> struct CpTileSel<128, 128> { using T = CpCfg<128, 128, 8, 16, 16, 4, 2>; };
template <> struct CpTileSel<128, 64> { using T = CpCfg<128, 64, 8, 8, 32, 3, 2>; };
template <> struct CpTileSel<64, 64> { using T = CpCfg<64, 64, 4, 8, 32, 3, 4>; };
// Grouped launches only, for problems of few rows: 4 x 8 outputs a thread over
// four by eight lanes, so a warp's B reads are whole 128-byte rows (the 74
// problems of at most 32 rows of a 128-GEMM batch, 2.3 GB of B: 0.54 ms; BK 16 x
// 4 stages and four CTAs an SM, or 16 x 128 tiles of 2 x 8 a thread, 0.93).
template <> struct CpTileSel<16, 256> { using T = CpCfg<16, 256, 4, 8, 32, 3, 2, 4>; };
template <int BM, int BN> using CpTile = typename CpTileSel<BM, BN>::T;

// Two FP32 lanes in a 64-bit register: the packed arithmetic of sm_100
// (fma.rn.f32x2), each lane rounded exactly as the scalar instruction rounds
// it.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// c + a * b: one fused multiply-add per lane, or (SCALAR variant) a multiply,
// then an add, each rounded. The latter is on single floats: the compiler
// contracts a packed multiply and add into the fused form (seen in results),
// which it never does to __fmul_rn and __fadd_rn.
__device__ __forceinline__ f32x2 mac(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float mac(float a, float b, float c) { return __fadd_rn(c, __fmul_rn(a, b)); }

// W floats from global to shared memory; with `bytes`, that many are read and
// the rest of the 4 W written as zeros.
template <int W>
__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, int bytes) {
    if constexpr (W == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"(dst), "l"(src), "r"(bytes), "n"(4 * W) : "memory");
}
template <int W>
__device__ __forceinline__ void cp_async(uint32_t dst, const float* src) {
    if constexpr (W == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(4 * W) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <class Cf, bool FUSED>
__device__ __forceinline__ void simt_cp_tile(const SimtArgs& p, int64_t m0, int64_t n0, int z, unsigned tile,
                                             float* smem, int& last_flag) {
    constexpr int BM = Cf::BM, BN = Cf::BN, BK = Cf::BK, STAGES = Cf::STAGES, THREADS = Cf::THREADS;
    constexpr int LT = Cf::LT, RT = Cf::RT;
    constexpr int AST = Cf::AST;
    constexpr int GN = LT / 4;                 // float4 groups per thread row
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp / Cf::WARPS_N, wn = warp % Cf::WARPS_N;
    const int lm = lane / Cf::LN, ln = lane % Cf::LN;
    const int64_t M = p.M, N = p.N, K = p.K;
    const int64_t kbeg = (int64_t)z * p.kchunk;
    const int64_t kend = min(K, kbeg + p.kchunk);
    const int64_t ntiles = (kend - kbeg + BK - 1) / BK;
    const float* __restrict__ A = p.A;
    const float* __restrict__ B = p.B;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);

    // Stage `buf` <- A[m0.., k0..k0+BK), B[k0..k0+BK, n0..) in copies of W
    // floats, the widest that every row start allows. A stage wholly inside the
    // slice and the matrix needs no bounds; otherwise copies outside read
    // nothing and write zeros (their source address is kept inside the operand).
    const bool inside = m0 + BM <= M && n0 + BN <= N;
    auto load_a_stage = [&]<int W, bool EDGE>(uint32_t a_s, int64_t k0) {
        constexpr int CPR = BK / W, RPP = THREADS / CPR;            // copies per row, rows per pass
        const int row = tid / CPR, col = tid % CPR * W;
        const float* src = A + (m0 + row) * K + k0 + col;
        const uint32_t dst = a_s + (uint32_t)(row * AST + col) * 4u;
        const int64_t step = (int64_t)RPP * K;
#pragma unroll(W == 1 ? 8 : 16)
        for (int j = 0; j < BM / RPP; j++, src += step) {
            if constexpr (EDGE) {
                const bool ok = k0 + col < kend && m0 + row + j * RPP < M;
                cp_async<W>(dst + (uint32_t)(j * RPP * AST * 4), ok ? src : A, ok ? 4 * W : 0);
            } else {
                cp_async<W>(dst + (uint32_t)(j * RPP * AST * 4), src);
            }
        }
    };
    auto load_b_stage = [&]<int W, bool EDGE>(uint32_t b_s, int64_t k0) {
        if constexpr (BN / W > THREADS) {                           // several copies of one row per thread
            for (int j = 0; j < BK; j++) {
                const float* src = B + (k0 + j) * N + n0;
#pragma unroll
                for (int col = 0; col < BN / W; col += THREADS) {
                    const int c = (col + tid) * W;
                    const bool ok = !EDGE || (k0 + j < kend && n0 + c < N);
                    cp_async<W>(b_s + (uint32_t)(j * BN + c) * 4u, ok ? src + c : B, ok ? 4 * W : 0);
                }
            }
            return;
        } else {
            constexpr int CPR = BN / W, RPP = THREADS / CPR;
            const int row = tid / CPR, col = tid % CPR * W;
            const float* src = B + (k0 + row) * N + n0 + col;
            const uint32_t dst = b_s + (uint32_t)(row * BN + col) * 4u;
            const int64_t step = (int64_t)RPP * N;
#pragma unroll(W == 1 ? 8 : 16)
            for (int j = 0; j < BK / RPP; j++, src += step) {
                if constexpr (EDGE) {
                    const bool ok = k0 + row + j * RPP < kend && n0 + col < N;
                    cp_async<W>(dst + (uint32_t)(j * RPP * BN * 4), ok ? src : B, ok ? 4 * W : 0);
                } else {
                    cp_async<W>(dst + (uint32_t)(j * RPP * BN * 4), src);
                }
            }
        }
    };
    auto load_stage = [&](int buf, int64_t k0) {
        const uint32_t a_s = sbase + (uint32_t)(buf * Cf::STAGE_FLOATS) * 4u;
        const uint32_t b_s = a_s + (uint32_t)Cf::A_FLOATS * 4u;
        if (inside && k0 + BK <= kend) {
            if (p.wa == 4) load_a_stage.template operator()<4, false>(a_s, k0);
            else if (p.wa == 2) load_a_stage.template operator()<2, false>(a_s, k0);
            else load_a_stage.template operator()<1, false>(a_s, k0);
            if (p.wb == 4) load_b_stage.template operator()<4, false>(b_s, k0);
            else if (p.wb == 2) load_b_stage.template operator()<2, false>(b_s, k0);
            else load_b_stage.template operator()<1, false>(b_s, k0);
        } else {
            if (p.wa == 4) load_a_stage.template operator()<4, true>(a_s, k0);
            else if (p.wa == 2) load_a_stage.template operator()<2, true>(a_s, k0);
            else load_a_stage.template operator()<1, true>(a_s, k0);
            if (p.wb == 4) load_b_stage.template operator()<4, true>(b_s, k0);
            else if (p.wb == 2) load_b_stage.template operator()<2, true>(b_s, k0);
            else load_b_stage.template operator()<1, true>(b_s, k0);
        }
    };

    // Packed pairs of outputs, or single ones in the SCALAR variant.
    using Elem = std::conditional_t<FUSED, f32x2, float>;
    using Quad = std::conditional_t<FUSED, ulonglong2, float4>;
    constexpr int NE = FUSED ? LT / 2 : LT, PER = NE / GN;
    Elem acc[RT][NE];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < NE; j++) acc[i][j] = 0;

    // Operand fragments of two k's: rows lm + 8 i of A, column quads of B.
    float2 fa[2][RT];
    Elem fb[2][NE];
    const int a_off = (wm * Cf::WM + lm) * AST, b_off = Cf::A_FLOATS + wn * Cf::WN + ln * 4;
    auto load_a = [&](int set, const float* st, int k) {
#pragma unroll
        for (int i = 0; i < RT; i++) fa[set][i] = *reinterpret_cast<const float2*>(st + a_off + i * Cf::LM * AST + k);
    };
    auto load_b = [&](int set, const float* st, int k) {
#pragma unroll
        for (int j = 0; j < GN; j++) {
            const Quad v = *reinterpret_cast<const Quad*>(st + b_off + k * BN + j * 4 * Cf::LN);
            fb[set][PER * j] = v.x;
            fb[set][PER * j + 1] = v.y;
            if constexpr (!FUSED) {
                fb[set][PER * j + 2] = v.z;
                fb[set][PER * j + 3] = v.w;
            }
        }
    };

#pragma unroll
    for (int st = 0; st < STAGES - 1; st++) {
        if (st < ntiles) load_stage(st, kbeg + (int64_t)st * BK);
        cp_async_commit();
    }
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    load_a(0, smem, 0);
    load_b(0, smem, 0);
    // Fragments of k + 1 are read while k's products run; the last k of a stage
    // reads the next stage's first ones, after the barrier that says that stage
    // has landed and that every warp has read the stage before it, whose buffer
    // the next copies take. (Past the last stage it reads a stale buffer, unused.)
    //
    // A stage is unrolled whole, or in the SCALAR variant, with four times the
    // instructions, four k's at a time: eight or sixteen are more code than the
    // instruction cache holds (sixty 128 x 128 plans, against an earlier kernel: four
    // k's 0.74 of its time on long K, eight 1.15, sixteen 1.43).
    constexpr int U = FUSED ? BK : 4;
    int buf = 0;
    for (int64_t t = 0; t < ntiles; t++) {
        const float* cur = smem + buf * Cf::STAGE_FLOATS;
        const int nbuf = buf + 1 == STAGES ? 0 : buf + 1;
        const float* nxt = smem + nbuf * Cf::STAGE_FLOATS;
#pragma unroll 1
        for (int k0 = 0; k0 < BK; k0 += U) {
#pragma unroll
            for (int k = 0; k < U; k++) {
                if (k + 1 < U || k0 + U < BK) {
                    load_b((k + 1) & 1, cur, k0 + k + 1);
                    if ((k & 1) == 1) load_a(((k + 1) >> 1) & 1, cur, k0 + k + 1);
                } else {
                    cp_async_wait<STAGES - 3>();
                    __syncthreads();
                    const int64_t tn = t + STAGES - 1;
                    if (tn < ntiles) load_stage(buf == 0 ? STAGES - 1 : buf - 1, kbeg + tn * BK);
                    cp_async_commit();
                    load_b(0, nxt, 0);
                    load_a(0, nxt, 0);
                }
                Elem aa[RT];
#pragma unroll
                for (int i = 0; i < RT; i++) {
                    const float2 v = fa[(k >> 1) & 1][i];
                    if constexpr (FUSED) aa[i] = (k & 1) ? pack2(v.y, v.y) : pack2(v.x, v.x);
                    else aa[i] = (k & 1) ? v.y : v.x;
                }
                // Column by column, rows down and up in turn: neighbouring
                // instructions share an operand.
#pragma unroll
                for (int j = 0; j < NE; j++)
#pragma unroll
                    for (int q = 0; q < RT; q++) {
                        const int i = (j & 1) ? RT - 1 - q : q;
                        acc[i][j] = mac(aa[i], fb[k & 1][j], acc[i][j]);
                    }
            }
        }
        buf = nbuf;
    }
    cp_async_wait<0>();

    // Steps past kend multiplied zeros: the chains are those over [kbeg, kend).
    float out[RT][LT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < NE; j++) {
            if constexpr (FUSED) unpack2(acc[i][j], out[i][2 * j], out[i][2 * j + 1]);
            else out[i][j] = acc[i][j];
        }
    auto out_row = [&](int i) { return m0 + wm * Cf::WM + lm + Cf::LM * i; };
    auto out_col = [&](int g) { return n0 + wn * Cf::WN + ln * 4 + 4 * Cf::LN * g; };
    simt_epilogue<RT, GN>(p, out, out_row, out_col, p.wc == 4, z, tile, last_flag);
}

template <class Cf, bool FUSED>
__global__ void __launch_bounds__(Cf::THREADS, Cf::CTAS)
sgemm_simt_cp_kernel(SimtArgs p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int last_flag;
    grid_wait();
    simt_cp_tile<Cf, FUSED>(p, (int64_t)blockIdx.y * Cf::BM, (int64_t)blockIdx.x * Cf::BN, blockIdx.z,
                            blockIdx.y * gridDim.x + blockIdx.x, smem, last_flag);
}

// ---------------------------------------------------------------------------
// The register-staged tile, for what the ring above is the slower at: the SCALAR
// variant on 64 columns, and short K slices.
//
// 256 threads, BM / 16 x BN / 16 outputs each; stages of 16 k's go through
// registers into two shared buffers, A transposed to k-major so that a fragment
// is read in 128-bit loads: As[k][m ^ (k & 8)], rows of BM + 4 floats, which keeps
// the transposing stores of a warp on distinct banks. Same chains, same bits.
//
// SCALAR: bound by the latency of multiply, then add, where a single wave leaves
// a warp or two a scheduler; this tile has two, and its unrolled stage fits the
// instruction cache. 1 x 10786 x 54 on 128 x 64 tiles 2466 us on the ring unrolled
// whole, 1199 in bodies of four k's, 958 here; over 120 plans 0.56-1.01 of the time
// of an earlier kernel by tile and K (geometric means), at most 1.03 of it.
// Short K: the ring's stage of 32 k's is loaded and multiplied whole, so K of 8 or
// 11 costs what 32 does: 1275 x 11 x 2921 on 128 x 64 tiles 14.4 -> 10.6 us, 3254 x 8 x 998
// on 64 x 64 12.1 -> 8.1. kShortK is where that stops paying for every tile; single
// launches go on to 31 k's on 64 x 64 tiles and 64 on 128 x 64, whose ring fills late
// (times over the ring's, geometric means: 17-32 k's 0.94 on 128 x 64, 1.01 on 64 x 64;
// 33-64 k's 0.97 and 1.04).
// ---------------------------------------------------------------------------
constexpr int kRegThreads = 256, RBK = 16;
constexpr int64_t kShortK = 16;

template <int BM, int BN>
struct RegSmem {
    float As[2][RBK][BM + 4];
    float Bs[2][RBK][BN];
};

template <bool FUSED>
__device__ __forceinline__ float reg_mac(float a, float b, float c) {
    if constexpr (FUSED) return __fmaf_rn(a, b, c);
    else return mac(a, b, c);
}

// VEC: 128-bit loads of A and B.
template <int BM, int BN, bool FUSED>
__device__ __forceinline__ void simt_reg_tile(const SimtArgs& p, int64_t m0, int64_t n0, int z, unsigned tile,
                                              RegSmem<BM, BN>& sm, int& last_flag, bool VEC) {
    constexpr int TM = BM / 16, TN = BN / 16;       // per-thread outputs
    constexpr int GM = TM / 4, GN = TN / 4;         // 4-wide groups per thread
    constexpr int A_F4 = BM * RBK / 4 / kRegThreads;   // float4 loads per thread
    constexpr int B_F4 = BN * RBK / 4 / kRegThreads;
    auto& As = sm.As;
    auto& Bs = sm.Bs;

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int64_t kbeg = (int64_t)z * p.kchunk;
    const int64_t kend = min(p.K, kbeg + p.kchunk);
    const int64_t M = p.M, N = p.N, K = p.K;
    const float* __restrict__ A = p.A;
    const float* __restrict__ B = p.B;

    float4 ra[A_F4], rb[B_F4];

    auto load_tile = [&](int64_t k0) {
#pragma unroll
        for (int j = 0; j < A_F4; j++) {
            const int f = tid + j * kRegThreads;
            const int row = f / (RBK / 4);
            const int kq = (f % (RBK / 4)) * 4;
            const int64_t gm = m0 + row, gk = k0 + kq;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (gm < M) {
                const float* src = A + gm * K + gk;
                if (VEC) {
                    if (gk < kend) v = __ldg(reinterpret_cast<const float4*>(src));
                } else {
                    if (gk + 0 < kend) v.x = __ldg(src + 0);
                    if (gk + 1 < kend) v.y = __ldg(src + 1);
                    if (gk + 2 < kend) v.z = __ldg(src + 2);
                    if (gk + 3 < kend) v.w = __ldg(src + 3);
                }
            }
            ra[j] = v;
        }
#pragma unroll
        for (int j = 0; j < B_F4; j++) {
            const int f = tid + j * kRegThreads;
            const int kr = f / (BN / 4);
            const int nq = (f % (BN / 4)) * 4;
            const int64_t gk = k0 + kr, gn = n0 + nq;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (gk < kend) {
                const float* src = B + gk * N + gn;
                if (VEC) {
                    if (gn < N) v = __ldg(reinterpret_cast<const float4*>(src));
                } else {
                    if (gn + 0 < N) v.x = __ldg(src + 0);
                    if (gn + 1 < N) v.y = __ldg(src + 1);
                    if (gn + 2 < N) v.z = __ldg(src + 2);
                    if (gn + 3 < N) v.w = __ldg(src + 3);
                }
            }
            rb[j] = v;
        }
    };
    auto store_tile = [&](int buf) {
#pragma unroll
        for (int j = 0; j < A_F4; j++) {
            const int f = tid + j * kRegThreads;
            const int row = f / (RBK / 4);
            const int kq = (f % (RBK / 4)) * 4;
            const int srow = row ^ (kq & 8);
            As[buf][kq + 0][srow] = ra[j].x;
            As[buf][kq + 1][srow] = ra[j].y;
            As[buf][kq + 2][srow] = ra[j].z;
            As[buf][kq + 3][srow] = ra[j].w;
        }
#pragma unroll
        for (int j = 0; j < B_F4; j++) {
            const int f = tid + j * kRegThreads;
            const int kr = f / (BN / 4);
            const int nq = (f % (BN / 4)) * 4;
            *reinterpret_cast<float4*>(&Bs[buf][kr][nq]) = rb[j];
        }
    };

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;

    const int64_t ntiles = (kend - kbeg + RBK - 1) / RBK;
    if (ntiles > 0) {
        load_tile(kbeg);
        store_tile(0);
        __syncthreads();
        for (int64_t t = 0; t < ntiles; t++) {
            const int buf = (int)(t & 1);
            if (t + 1 < ntiles) load_tile(kbeg + (t + 1) * RBK);
            // Fragments of step k + 1 are read from shared memory while the
            // products of step k run (two register sets, fully unrolled).
            float a[2][TM], b[2][TN];
            auto load_frag = [&](int set, int k) {
#pragma unroll
                for (int g = 0; g < GM; g++) {
                    float4 v = *reinterpret_cast<const float4*>(&As[buf][k][(g * 64 + ty * 4) ^ (k & 8)]);
                    a[set][g * 4 + 0] = v.x; a[set][g * 4 + 1] = v.y; a[set][g * 4 + 2] = v.z; a[set][g * 4 + 3] = v.w;
                }
#pragma unroll
                for (int g = 0; g < GN; g++) {
                    float4 v = *reinterpret_cast<const float4*>(&Bs[buf][k][g * 64 + tx * 4]);
                    b[set][g * 4 + 0] = v.x; b[set][g * 4 + 1] = v.y; b[set][g * 4 + 2] = v.z; b[set][g * 4 + 3] = v.w;
                }
            };
            load_frag(0, 0);
#pragma unroll
            for (int k = 0; k < RBK; k++) {
                // A short K stops after its last four k's.
                if (FUSED && k > 0 && k % 4 == 0 && kbeg + t * RBK + k >= kend) break;
                if (k + 1 < RBK) load_frag((k + 1) & 1, k + 1);
#pragma unroll
                for (int i = 0; i < TM; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) acc[i][j] = reg_mac<FUSED>(a[k & 1][i], b[k & 1][j], acc[i][j]);
            }
            if (t + 1 < ntiles) store_tile(buf ^ 1);
            __syncthreads();
        }
    }

    // Steps past kend multiplied zeros, as above.
    auto out_row = [&](int i) { return m0 + (i / 4) * 64 + ty * 4 + (i % 4); };
    auto out_col = [&](int g) { return n0 + g * 64 + tx * 4; };
    simt_epilogue<TM, GN>(p, acc, out_row, out_col, p.wc == 4, z, tile, last_flag);
}

template <int BM, int BN, bool FUSED, bool VEC>
__global__ void __launch_bounds__(kRegThreads, 2)
sgemm_simt_reg_kernel(SimtArgs p) {
    __shared__ __align__(16) RegSmem<BM, BN> sm;
    __shared__ int last_flag;
    grid_wait();
    simt_reg_tile<BM, BN, FUSED>(p, (int64_t)blockIdx.y * BM, (int64_t)blockIdx.x * BN, blockIdx.z,
                                 blockIdx.y * gridDim.x + blockIdx.x, sm, last_flag, VEC);
}

// Grouped launch: one persistent kernel over a list of (problem, tile, K
// slice) units taken from an atomic counter, heaviest units first. Each unit
// is exactly the tile a per-GEMM launch of that problem computes, so results
// are identical to running the problems one by one.
template <class RunUnit>
__device__ __forceinline__ void grouped_units(const GroupProblem* __restrict__ probs, const GroupUnit* __restrict__ units,
                                              int nunits, unsigned* next, RunUnit run) {
    __shared__ int s_unit;
    grid_wait();
    // Thread 0 fetches the next unit's number while the current one runs.
    unsigned fetched = threadIdx.x == 0 ? atomicAdd(next, 1u) : 0u;
    for (;;) {
        if (threadIdx.x == 0) s_unit = (int)min(fetched, (unsigned)nunits);
        __syncthreads();                     // also: the last unit's stages are no longer read
        const int u = s_unit;
        if (u >= nunits) break;
        if (threadIdx.x == 0) fetched = atomicAdd(next, 1u);
        const GroupUnit w = units[u];
        const GroupProblem& P = probs[w.problem];
        const unsigned tile = (unsigned)w.tm * (unsigned)P.tiles_n + (unsigned)w.tn;
        run(P.a, w, tile);
    }
}

template <class Cf, bool FUSED>
__global__ void __launch_bounds__(Cf::THREADS, Cf::CTAS)
sgemm_simt_grouped_kernel(const GroupProblem* __restrict__ probs, const GroupUnit* __restrict__ units, int nunits,
                          unsigned* next) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int last_flag;
    grouped_units(probs, units, nunits, next, [&](const SimtArgs& args, const GroupUnit& w, unsigned tile) {
        const SimtArgs a = args;
        simt_cp_tile<Cf, FUSED>(a, (int64_t)w.tm * Cf::BM, (int64_t)w.tn * Cf::BN, w.z, tile, smem, last_flag);
    });
}

template <int BM, int BN, bool FUSED>
__global__ void __launch_bounds__(kRegThreads, 2)
sgemm_simt_reg_grouped_kernel(const GroupProblem* __restrict__ probs, const GroupUnit* __restrict__ units, int nunits,
                              unsigned* next) {
    __shared__ __align__(16) RegSmem<BM, BN> sm;
    __shared__ int last_flag;
    grouped_units(probs, units, nunits, next, [&](const SimtArgs& a, const GroupUnit& w, unsigned tile) {
        simt_reg_tile<BM, BN, FUSED>(a, (int64_t)w.tm * BM, (int64_t)w.tn * BN, w.z, tile, sm, last_flag,
                                     a.wa == 4 && a.wb == 4);
    });
}

// Split-K reduction of the single launches (grouped launches sum in the last
// CTA of a tile to arrive, simt_epilogue): the slices wrote their partial
// products ([slice][M][N]); each thread sums one output (T =
// float) or four adjacent ones (T = float4) over the slices in slice order --
// the order of the in-kernel fixup and of the reference's panel sum
// C = p0 + p1 + ... -- so C is the same bit for bit. Two slices go this way too:
// clearing and counting arrivals costs more than the second launch (128 x 64
// tiles, two slices: 2048^3 344 -> 331 us, 1024^3 62 -> 53, 300^3 29 -> 13). Bound by the reads of the
// partials, splits * M * N floats, from L2 while they fit (126 MB). Measured
// (ncu): 1024^2 x 8 slices 7.8-9.2 us by run (4.1-4.8 TB/s), 777 x 901 x 8 6.3 us, 512^2 x 16
// 5.4 us, 256^2 x 8 3.1 us; a grid-stride loop with a fixed batch of 64
// predicated evict-first loads took 50, 36, 16.4 and 5.7 us.
template <int BATCH, typename T>
__global__ void __launch_bounds__(256)
simt_splitk_reduce_kernel(const T* __restrict__ partial, T* __restrict__ C, int64_t n, int splits) {
    grid_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) C[i] = ordered_sum<BATCH>(partial + i, (size_t)n, splits);
}

template <typename T>
cudaError_t launch_splitk_reduce(const float* partial, float* C, int64_t n, int splits, cudaStream_t s) {
    const unsigned blocks = (unsigned)((n + 255) / 256);
    const T* src = reinterpret_cast<const T*>(partial);
    T* dst = reinterpret_cast<T*>(C);
    auto kernel = splits <= 4 ? simt_splitk_reduce_kernel<3, T> : splits <= 8 ? simt_splitk_reduce_kernel<7, T>
                : sizeof(T) > 4 || splits <= 16 ? simt_splitk_reduce_kernel<15, T>
                                                : simt_splitk_reduce_kernel<(sizeof(T) > 4 ? 15 : 63), T>;
    return launch_overlapped(kernel, dim3(blocks), 256, 0, s, 1, src, dst, n, splits);
}

// Four outputs per thread where rows of four stay 16-byte aligned in every
// slice and the quads alone give the GPU enough threads (two blocks an SM:
// 1024^2 has 1024 blocks of quads); a small C keeps one output per thread and
// has up to 63 slices in flight at once, since its loads wait for latency, not
// bandwidth (64 x 512 x 64 slices: 4.8 us on 128 blocks).
cudaError_t splitk_reduce(const SimtArgs& a, cudaStream_t s) {
    const int64_t n = a.M * a.N;
    if (n % 4 == 0 && (uintptr_t)a.C % 16 == 0 && n / 4 >= (int64_t)device_sm_count() * 512)
        return launch_splitk_reduce<float4>(a.partial, a.C, n / 4, a.splits, s);
    return launch_splitk_reduce<float>(a.partial, a.C, n, a.splits, s);
}

// Raises a kernel's dynamic shared memory limit once per device.
template <typename Kern>
cudaError_t smem_limit_once(Kern kern, int bytes, std::atomic<uint64_t>& done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && ((done.load() >> dev) & 1u)) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
    return e;
}

template <class Cf, bool FUSED>
cudaError_t launch_cp(const SimtArgs& a, dim3 grid, cudaStream_t s) {
    static std::atomic<uint64_t> done{0};
    cudaError_t e = smem_limit_once(sgemm_simt_cp_kernel<Cf, FUSED>, Cf::SMEM, done);
    if (e != cudaSuccess) return e;
    return launch_overlapped(sgemm_simt_cp_kernel<Cf, FUSED>, grid, Cf::THREADS, Cf::SMEM, s, 1, a);
}

template <int BM, int BN, bool FUSED>
cudaError_t launch_reg(const SimtArgs& a, dim3 grid, cudaStream_t s) {
    auto kernel = a.wa == 4 && a.wb == 4 ? sgemm_simt_reg_kernel<BM, BN, FUSED, true> : sgemm_simt_reg_kernel<BM, BN, FUSED, false>;
    return launch_overlapped(kernel, grid, kRegThreads, 0, s, 1, a);
}

template <int BM, int BN>
cudaError_t launch_tile(const SimtArgs& args, int variant, cudaStream_t s) {
    using Cf = CpTile<BM, BN>;
    const bool scalar = variant == MAXMULSK_FP32_SCALAR;
    SimtArgs a = args;
    a.reduce_after = a.splits > 1 ? 1 : 0;
    simt_set_widths(a);
    const dim3 grid((unsigned)((a.N + BN - 1) / BN), (unsigned)((a.M + BM - 1) / BM), (unsigned)a.splits);
    cudaError_t e;
    {
        PhaseScope ps(kPhaseGemm, s);
        if constexpr (BN == 64) {
            if (scalar) e = launch_reg<BM, BN, false>(a, grid, s);
            else if (std::min(a.K, a.kchunk) <= (BM == 128 ? 64 : 31)) e = launch_reg<BM, BN, true>(a, grid, s);
            else e = launch_cp<Cf, true>(a, grid, s);
        } else {
            e = scalar ? launch_cp<Cf, false>(a, grid, s) : launch_cp<Cf, true>(a, grid, s);
        }
    }
    if (e != cudaSuccess || !a.reduce_after) return e;
    PhaseScope ps(kPhaseReduce, s);
    return splitk_reduce(a, s);
}

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

size_t simt_workspace_bytes(int64_t M, int64_t K, int64_t N, int tile_m, int tile_n, int split_k) {
    const int splits = slice_count((size_t)K, split_k);
    if (splits <= 1) return 0;
    const size_t tiles = (size_t)((M + tile_m - 1) / tile_m) * (size_t)((N + tile_n - 1) / tile_n);
    return align256(tiles * sizeof(unsigned)) + align256((size_t)splits * (size_t)M * (size_t)N * sizeof(float));
}

bool simt_bind_workspace(SimtArgs& a, int tile_m, int tile_n, void* ws, size_t ws_bytes) {
    if (a.splits <= 1) { a.partial = nullptr; a.counters = nullptr; return true; }
    const size_t tiles = (size_t)((a.M + tile_m - 1) / tile_m) * (size_t)((a.N + tile_n - 1) / tile_n);
    const size_t need = align256(tiles * sizeof(unsigned)) + align256((size_t)a.splits * a.M * a.N * sizeof(float));
    if (!ws || ws_bytes < need) return false;
    a.counters = static_cast<unsigned*>(ws);
    a.partial = reinterpret_cast<float*>(static_cast<char*>(ws) + align256(tiles * sizeof(unsigned)));
    return true;
}

cudaError_t simt_launch(const SimtArgs& a, int tile_m, int tile_n, int variant, cudaStream_t s) {
    if (tile_m == 128 && tile_n == 128) return launch_tile<128, 128>(a, variant, s);
    if (tile_m == 128 && tile_n == 64) return launch_tile<128, 64>(a, variant, s);
    if (tile_m == 64 && tile_n == 64) return launch_tile<64, 64>(a, variant, s);
    return cudaErrorInvalidValue;
}

maxmulsk_status simt_run(const float* dA, const float* dB, float* dC, size_t M, size_t K, size_t N,
                         const maxmulsk_plan& plan, void* scratch, size_t scratch_bytes, cudaStream_t s) {
    SimtArgs a{};
    a.A = dA; a.B = dB; a.C = dC;
    a.M = (int64_t)M; a.K = (int64_t)K; a.N = (int64_t)N;
    a.kchunk = (int64_t)slice_len(K, plan.split_k);
    a.splits = slice_count(K, plan.split_k);
    if (!simt_bind_workspace(a, plan.tile_m, plan.tile_n, scratch, scratch_bytes)) {
        set_error_message("workspace too small for the SIMT plan");
        return MAXMULSK_ERR_INVALID;
    }
    return cuda_status(simt_launch(a, plan.tile_m, plan.tile_n, plan.variant, s), "sgemm_simt launch");
}

namespace {
template <class Cf, bool FUSED>
cudaError_t launch_grouped(const GroupProblem* probs, const GroupUnit* units, int nunits, unsigned* next, int sms,
                           cudaStream_t s) {
    static std::atomic<uint64_t> done{0};
    cudaError_t e = smem_limit_once(sgemm_simt_grouped_kernel<Cf, FUSED>, Cf::SMEM, done);
    if (e != cudaSuccess) return e;
    const int slots = Cf::CTAS * sms;
    return launch_overlapped(sgemm_simt_grouped_kernel<Cf, FUSED>, dim3(nunits < slots ? nunits : slots), Cf::THREADS,
                             Cf::SMEM, s, 1, probs, units, nunits, next);
}
template <int BM, int BN, bool FUSED>
cudaError_t launch_reg_grouped(const GroupProblem* probs, const GroupUnit* units, int nunits, unsigned* next, int sms,
                               cudaStream_t s) {
    return launch_overlapped(sgemm_simt_reg_grouped_kernel<BM, BN, FUSED>, dim3(std::min(nunits, 2 * sms)), kRegThreads, 0, s, 1,
                             probs, units, nunits, next);
}
template <int BM, int BN>
cudaError_t launch_grouped_tile(const GroupProblem* probs, const GroupUnit* units, int nunits, unsigned* next,
                                int variant, int sms, int64_t longest, cudaStream_t s) {
    using Cf = CpTile<BM, BN>;
    const bool scalar = variant == MAXMULSK_FP32_SCALAR;
    if constexpr (BM >= 64) {
        if (scalar && (BN == 64 || longest <= kShortK)) return launch_reg_grouped<BM, BN, false>(probs, units, nunits, next, sms, s);
        if (!scalar && longest <= kShortK) return launch_reg_grouped<BM, BN, true>(probs, units, nunits, next, sms, s);
    }
    if constexpr (BN != 64)
        if (scalar) return launch_grouped<Cf, false>(probs, units, nunits, next, sms, s);
    return launch_grouped<Cf, true>(probs, units, nunits, next, sms, s);
}
}  // namespace

cudaError_t simt_grouped_launch(const GroupProblem* probs, const GroupUnit* units, int nunits, unsigned* next,
                                int tile_m, int tile_n, int variant, int sms, int64_t longest, cudaStream_t s) {
    if (tile_m == 128 && tile_n == 128) return launch_grouped_tile<128, 128>(probs, units, nunits, next, variant, sms, longest, s);
    if (tile_m == 128 && tile_n == 64) return launch_grouped_tile<128, 64>(probs, units, nunits, next, variant, sms, longest, s);
    if (tile_m == 64 && tile_n == 64) return launch_grouped_tile<64, 64>(probs, units, nunits, next, variant, sms, longest, s);
    if (tile_m == 16 && tile_n == 256) return launch_grouped_tile<16, 256>(probs, units, nunits, next, variant, sms, longest, s);
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Static-scratch variant: the split-K SIMT path with its counters and partial
// tiles in a fixed device array instead of caller or library allocations.
//
// Some callers cannot allocate device memory at the point of the call: a
// host application that owns the whole device memory budget and forbids its
// plug-ins to call cudaMalloc, or a latency-critical loop that cannot afford
// cudaMalloc/cudaFree (which may synchronise the device). For them this path
// allocates nothing: the scratch lives in the array below, which the module
// reserves on every GPU that loads this library and keeps until the process
// exits.
//
// Limits and rules:
//   * at most MAXMULSK_STATIC_SCRATCH_BYTES (16 MiB) of scratch: a plan that
//     needs more is rejected (MAXMULSK_ERR_UNSUPPORTED), C untouched;
//   * one array per device, shared by every call: calls that overlap on the
//     GPU (other streams, other host threads) race on it and must be
//     serialised by the caller;
//   * the first call on a device resolves the array's device address
//     (cudaGetSymbolAddress) with that device current; make that first call
//     before any stream capture. The address is kept per CUDA context, so a
//     context made after cudaDeviceReset resolves it again (its first call,
//     too, belongs before any capture);
//   * the array keeps the last call's contents; every launch writes what it
//     reads.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_simt_static_scratch[MAXMULSK_STATIC_SCRATCH_BYTES];

namespace {

// The array's device address is resolved once per CUDA context (the primary
// context of each device the library is used on), keyed on the context's
// process-unique id (cuCtxGetId), so a context created after cudaDeviceReset
// resolves it again instead of reusing an address that no longer exists.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

struct StaticAddr {
    int device;
    unsigned long long ctx_id;
    void* ptr;
};
std::mutex g_static_mu;
std::vector<StaticAddr> g_static_addr;

template <typename Fn>
Fn driver_fn(const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
        return reinterpret_cast<Fn>(p);
    return nullptr;
}

// Id of the current context (0 when the driver cannot say, which then keys
// the cache on the device alone).
unsigned long long current_context_id() {
    static CtxGetCurrentFn get_ctx = driver_fn<CtxGetCurrentFn>("cuCtxGetCurrent");
    static CtxGetIdFn get_id = driver_fn<CtxGetIdFn>("cuCtxGetId");
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_ctx && get_id && get_ctx(&c) == CUDA_SUCCESS && c && get_id(c, &id) == CUDA_SUCCESS) return id;
    return 0;
}

// Device address of g_simt_static_scratch in the current context. A thread
// with no context bound yet (id 0) resolves the address, which binds the
// device's primary context, and records it under that context's id.
cudaError_t static_scratch_address(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (ctx != 0)
        for (const StaticAddr& a : g_static_addr)
            if (a.device == dev && a.ctx_id == ctx) { *out = a.ptr; return cudaSuccess; }
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_simt_static_scratch);
    if (e != cudaSuccess) return e;
    ctx = current_context_id();
    for (StaticAddr& a : g_static_addr)
        if (a.device == dev) { a.ctx_id = ctx; a.ptr = p; *out = p; return cudaSuccess; }
    g_static_addr.push_back(StaticAddr{dev, ctx, p});
    *out = p;
    return cudaSuccess;
}

}  // namespace

maxmulsk_status simt_run_static_scratch(const float* dA, const float* dB, float* dC, size_t M, size_t K, size_t N,
                                        const maxmulsk_plan& plan, cudaStream_t s) {
    maxmulsk_status st = classify_plan(M, K, N, &plan);
    if (st != MAXMULSK_OK) return st;
    if (plan.precision != MAXMULSK_PREC_FP32) {
        set_error_message("the static-scratch entry runs FP32 plans only");
        return MAXMULSK_ERR_UNSUPPORTED;
    }
    if (handle_empty_dev(dC, M, K, N, s, &st)) return st;
    if (!dA || !dB || !dC) { set_error_message("null matrix pointer"); return MAXMULSK_ERR_INVALID; }
    const size_t need = simt_workspace_bytes((int64_t)M, (int64_t)K, (int64_t)N, plan.tile_m, plan.tile_n, plan.split_k);
    if (need > (size_t)MAXMULSK_STATIC_SCRATCH_BYTES) {
        set_error_message("plan needs more scratch than the static maximum of MAXMULSK_STATIC_SCRATCH_BYTES (16 MiB)");
        return MAXMULSK_ERR_UNSUPPORTED;
    }
    void* base = nullptr;
    if (need > 0) {
        st = cuda_status(static_scratch_address(&base), "cudaGetSymbolAddress(static scratch)");
        if (st != MAXMULSK_OK) return st;
    }
    return simt_run(dA, dB, dC, M, K, N, plan, base, need, s);
}

}  // namespace mmsk
