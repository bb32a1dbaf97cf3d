// TMA-fed variant of the f64 / Complex64 DMMA contraction (included by contract_dmma.cu).
//
// When each of M, N, K is a single fused mode and one side of every operand has unit stride,
// the operand tiles need no per-thread gather: one thread at a time issues two cp.async.bulk.tensor
// loads per k-iteration, one to six iterations ahead, and the CTA's four to sixteen warps do nothing
// else but fragment loads and DMMAs, synchronised by full/empty mbarriers (no CTA-wide barrier in
// the main loop, and the ring keeps running across the tiles of a stream-K range).
//
// The tensor maps are built so that the box lands in the order the m16n8k8 fragments are
// read, which makes every fragment load conflict-free without padding:
//   K-major operand   [k-panel of 4][row][4 k]     one 64-byte (complex) / 32-byte (real) run per row
//   MN-major operand  [row-group][k][G rows]       G = 2 (complex) or 4 (real): 32-byte runs
// (a quarter warp of 16-byte loads, or a half warp of 8-byte loads, then covers one
// contiguous 128-byte line).  Both are ordinary rank-4 tensor maps over the strided operand:
// dimension 0 is the short run, and a second dimension walks the same index in steps of the
// run length, which therefore has to divide the extent.
//
// The four-product complex form takes any extent.  A complex element is 16 bytes, all that TMA asks of
// an address, so dimension 0 can be the whole extent (zero-filled past its end) with one load per
// run.  To keep those few, runs are 128-byte lines:
//   K-major   [k-panel of 8][row][8 k]    one load per 8 k
//   MN-major  [group of 8 rows][k][8 rows]    8 loads for 64 rows (one load where 8 divides the extent)
// with TMA's 128-byte swizzle; lane (row r, slot c) reads k = 2c and 2c + 1 of an 8-deep step, so a
// quarter warp (two rows, four k of one parity) finds its 16-byte units in chunks (r ^ k) mod 8 that take
// every value once.  (Which k meets which slot of an MMA does not matter while both operands agree.)
// The issue of ten loads is nothing next to the 8000 clocks of a k-iteration's MMAs.  Such extents - odd
// bond dimensions - used to be left to the gather kernel: a chain with chi = 97 took 18.5 + 10.5 us
// (kernel and fix-up launch) per product, 9.8 us here.
#pragma once
#include "f64_map.h"
#include "ptx_sm100.cuh"

namespace tfb {

// FOUR (complex only): four real products per complex one, each part accurate to its own size.
template <bool CPLX, int BM_, int BN_, int BK_, int WARPS_M_, int WARPS_N_, int STAGES_, bool FOUR = false>
struct DmmaTmaCfg {
    using Base = DmmaCfg<CPLX, BM_, BN_, BK_, WARPS_M_, WARPS_N_, STAGES_>;  // tile shape, fix-up kernel
    static constexpr bool kCplx = CPLX, kFour = FOUR;
    static constexpr int ACC = CPLX ? (FOUR ? 4 : 6) : 2;  // accumulators per fragment element pair
    static constexpr int BM = BM_, BN = BN_, BK = BK_, WARPS_M = WARPS_M_, WARPS_N = WARPS_N_, STAGES = STAGES_;
    static constexpr int CONSUMERS = WARPS_M * WARPS_N;
    static constexpr int NT = CONSUMERS * 32;
    static constexpr int WM = BM / WARPS_M, WN = BN / WARPS_N;
    static constexpr int TM = WM / 8, TN = WN / 8;
    static constexpr int ES = CPLX ? 16 : 8;
    static constexpr bool kLines = FOUR;             // 128-byte runs, swizzled
    static constexpr int KR = kLines ? 8 : 4;        // k per run of a K-major tile
    static constexpr int G = kLines ? 8 : CPLX ? 2 : 4;  // rows per run of an MN-major tile
    static constexpr int A_BYTES = BM * BK * ES, B_BYTES = BN * BK * ES;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 16 * STAGES + 16 + 1024;
    static_assert(BM * BN * ES <= STAGES * STAGE_BYTES, "a tile's sums fit the ring");
};

// Element offset of (row, k) inside a dense tile.
template <typename Cfg, int ROWS, bool MN>
__device__ __forceinline__ int tile_off(int row, int k) {
    if (MN) return ((row / Cfg::G) * Cfg::BK + k) * Cfg::G + (row % Cfg::G);
    return ((k >> 2) * ROWS + row) * 4 + (k & 3);
}

// A lane's 16-byte units of a complex tile: row w0 + 8 i + lr, k = kk + 2 lc + q (kk a multiple of 8).  What
// depends on the lane is computed here, once; the rest of an address is a constant.
template <typename Cfg, int ROWS, bool MN>
struct LineReader {
    const char* at[2];
    __device__ __forceinline__ LineReader(const char* tile, int w0, int lr, int lc) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int k = 2 * lc + q;
            at[q] = tile + (MN ? w0 * (Cfg::BK * 16) + k * 128 : (w0 + lr) * 128) + ((lr ^ k) << 4);
        }
    }
    __device__ __forceinline__ double2 get(int i, int kk, int q) const {
        return *reinterpret_cast<const double2*>(at[q] + (MN ? i * Cfg::BK * 128 + kk * 128 : kk * ROWS * 16 + i * 1024));
    }
};

__device__ __forceinline__ double flip_sign(double x, unsigned mask) {
    return __hiloint2double((int)((unsigned)__double2hiint(x) ^ mask), __double2loint(x));
}

template <typename Cfg, bool A_MN, bool B_MN>
__device__ __forceinline__ void dmma_tma_consume(const char* sa, const char* sb, double (&acc)[Cfg::TM][Cfg::TN][Cfg::ACC],
                                                 int wm0, int wn0, int lr, int lc, bool conj_a, bool conj_b) {
    [[maybe_unused]] const double sign_a = conj_a ? -1.0 : 1.0, sign_b = conj_b ? -1.0 : 1.0;
    [[maybe_unused]] const unsigned flip_a = conj_a ? 0x80000000u : 0u, flip_b = conj_b ? 0x80000000u : 0u;
    constexpr bool CPLX = Cfg::kCplx;
    constexpr int TM = Cfg::TM, TN = Cfg::TN;
#pragma unroll
    for (int kk = 0; kk < Cfg::BK; kk += 8) {
        if constexpr (Cfg::kFour) {
            // Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br; acc[..][0..1] = Re, [2..3] = Im.
            const LineReader<Cfg, Cfg::BM, A_MN> ra(sa, wm0, lr, lc);
            const LineReader<Cfg, Cfg::BN, B_MN> rb(sb, wn0, lr, lc);
            double ar[TM][2], ai[TM][2], br[TN][2], bi[TN][2], nbi[TN][2];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v = ra.get(i, kk, q);
                    ar[i][q] = v.x;
                    ai[i][q] = flip_sign(v.y, flip_a);
                }
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v = rb.get(j, kk, q);
                    br[j][q] = v.x;
                    bi[j][q] = flip_sign(v.y, flip_b);
                    nbi[j][q] = flip_sign(v.y, flip_b ^ 0x80000000u);
                }
            auto pass = [&](const double (&x)[TM][2], const double (&y)[TN][2], int at) {
#pragma unroll
                for (int i = 0; i < TM; i += 2)
#pragma unroll
                    for (int j = 0; j < TN; ++j)
                        dmma16(acc[i][j][at], acc[i][j][at + 1], acc[i + 1][j][at], acc[i + 1][j][at + 1], x[i][0], x[i + 1][0],
                               x[i][1], x[i + 1][1], y[j][0], y[j][1]);
            };
            pass(ar, br, 0);
            pass(ar, bi, 2);
            pass(ai, nbi, 0);
            pass(ai, br, 2);
        } else if constexpr (CPLX) {
            // Three real products per complex one instead of four:
            //   P1 = Ar Br,  P2 = Ai Bi,  P3 = (Ar + Ai)(Br + Bi);  Re = P1 - P2,  Im = P3 - P1 - P2.
            // The sums cost two FMAs per fragment element; the FP64 pipe, which is what this
            // kernel waits for, issues a quarter fewer MMAs.  acc[..][0..1] = P1, [2..3] = P2,
            // [4..5] = P3; the caller folds them into Re / Im when a k range ends.  Conjugation is a sign in the sums
            // and, for P2, the caller's: everything but MMAs in this loop is time that the pipe stands still.
            double ar[TM][2], ai[TM][2], as[TM][2], br[TN][2], bi[TN][2], bs[TN][2];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v = *reinterpret_cast<const double2*>(
                        sa + (size_t)tile_off<Cfg, Cfg::BM, A_MN>(wm0 + 8 * i + lr, kk + 4 * q + lc) * 16);
                    ar[i][q] = v.x;
                    ai[i][q] = v.y;
                    as[i][q] = fma(sign_a, v.y, v.x);
                }
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v = *reinterpret_cast<const double2*>(
                        sb + (size_t)tile_off<Cfg, Cfg::BN, B_MN>(wn0 + 8 * j + lr, kk + 4 * q + lc) * 16);
                    br[j][q] = v.x;
                    bi[j][q] = v.y;
                    bs[j][q] = fma(sign_b, v.y, v.x);
                }
#pragma unroll
            for (int i = 0; i < TM; i += 2)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    dmma16(acc[i][j][0], acc[i][j][1], acc[i + 1][j][0], acc[i + 1][j][1], ar[i][0], ar[i + 1][0], ar[i][1],
                           ar[i + 1][1], br[j][0], br[j][1]);
#pragma unroll
            for (int i = 0; i < TM; i += 2)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    dmma16(acc[i][j][2], acc[i][j][3], acc[i + 1][j][2], acc[i + 1][j][3], ai[i][0], ai[i + 1][0], ai[i][1],
                           ai[i + 1][1], bi[j][0], bi[j][1]);
#pragma unroll
            for (int i = 0; i < TM; i += 2)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    dmma16(acc[i][j][4], acc[i][j][5], acc[i + 1][j][4], acc[i + 1][j][5], as[i][0], as[i + 1][0], as[i][1],
                           as[i + 1][1], bs[j][0], bs[j][1]);
        } else {
            double af[TM][2], bf[TN][2];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    af[i][q] = *reinterpret_cast<const double*>(
                        sa + (size_t)tile_off<Cfg, Cfg::BM, A_MN>(wm0 + 8 * i + lr, kk + 4 * q + lc) * 8);
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    bf[j][q] = *reinterpret_cast<const double*>(
                        sb + (size_t)tile_off<Cfg, Cfg::BN, B_MN>(wn0 + 8 * j + lr, kk + 4 * q + lc) * 8);
#pragma unroll
            for (int i = 0; i < TM; i += 2)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    dmma16(acc[i][j][0], acc[i][j][1], acc[i + 1][j][0], acc[i + 1][j][1], af[i][0], af[i + 1][0], af[i][1],
                           af[i + 1][1], bf[j][0], bf[j][1]);
        }
    }
}

// Element `t` (a thread of the main kernel) of fragment f = (i, j, e) of the tile at (m0, n0), finished and stored.
template <typename Cfg>
__device__ __forceinline__ void dmma_tma_store_one(const ContractArgs& g, int64_t bb, int64_t m0, int64_t n0, int f, int t, double xr,
                                                   double xi) {
    constexpr bool CPLX = Cfg::kCplx;
    const int i = f / (2 * Cfg::TN), j = (f >> 1) % Cfg::TN, e = f & 1, lane = t & 31, warp = t >> 5;
    const int64_t m = m0 + (warp % Cfg::WARPS_M) * Cfg::WM + 8 * i + (lane >> 2);
    const int64_t n = n0 + (warp / Cfg::WARPS_M) * Cfg::WN + 8 * j + 2 * (lane & 3) + e;
    if (m >= g.M || n >= g.N) return;
    if (g.mul) {
        const int64_t off = g.off_d_b(bb) + g.off_d_m(m) + g.off_d_n(n);
        if (CPLX) apply_mul_c128(g, off, xr, xi);
        else apply_mul_f64(g, off, xr);
    }
    dmma_store<CPLX>(g, g.c + (g.off_c_b(bb) + g.off_c_m(m) + g.off_c_n(n)) * (int64_t)Cfg::ES, g.beta_re != 0.0 || g.beta_im != 0.0, xr,
                     xi);
}

// Scratch slot of CTA `c` for a range that starts inside its tile (kind 0) or starts its tile (kind 1).
template <typename Cfg>
__device__ __forceinline__ char* dmma_tma_slot(const ContractArgs& g, int kind, int64_t c) {
    return g.partial + (size_t)(kind * (int64_t)gridDim.x + c) * (Cfg::BM * Cfg::BN) * Cfg::ES;
}
template <typename Cfg>
__device__ __forceinline__ void dmma_tma_park(char* P, const double (&acc)[Cfg::TM][Cfg::TN][Cfg::ACC], int tid) {
#pragma unroll
    for (int i = 0; i < Cfg::TM; ++i)
#pragma unroll
        for (int j = 0; j < Cfg::TN; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                char* q = P + ((size_t)((i * Cfg::TN + j) * 2 + e) * Cfg::NT + tid) * Cfg::ES;
                if constexpr (Cfg::kCplx) *reinterpret_cast<double2*>(q) = make_double2(acc[i][j][e], acc[i][j][2 + e]);
                else *reinterpret_cast<double*>(q) = acc[i][j][e];
            }
}
// A slot added to acc (ADD), or in its place.
template <typename Cfg, bool ADD>
__device__ __forceinline__ void dmma_tma_gather(const char* P, double (&acc)[Cfg::TM][Cfg::TN][Cfg::ACC], int tid) {
#pragma unroll
    for (int i = 0; i < Cfg::TM; ++i)
#pragma unroll
        for (int j = 0; j < Cfg::TN; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const char* q = P + ((size_t)((i * Cfg::TN + j) * 2 + e) * Cfg::NT + tid) * Cfg::ES;
                if constexpr (Cfg::kCplx) {
                    const double2 v = __ldcg(reinterpret_cast<const double2*>(q));
                    acc[i][j][e] = ADD ? acc[i][j][e] + v.x : v.x;
                    acc[i][j][2 + e] = ADD ? acc[i][j][2 + e] + v.y : v.y;
                } else {
                    const double v = __ldcg(reinterpret_cast<const double*>(q));
                    acc[i][j][e] = ADD ? acc[i][j][e] + v : v;
                }
            }
}

template <typename Cfg>
__global__ void __launch_bounds__(Cfg::NT, 1)
contract_dmma_tma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         ContractArgs g, int* status) {
    constexpr bool CPLX = Cfg::kCplx;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, TM = Cfg::TM, TN = Cfg::TN, STAGES = Cfg::STAGES;
    constexpr int ES = Cfg::ES;
    extern __shared__ __align__(128) char smem_dyn[];
    char* smem = (char*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);  // the swizzle follows address bits
    const uint32_t ring = smem_u32(smem);
    const uint32_t bars = ring + STAGES * Cfg::STAGE_BYTES;
    auto bar_full = [&](int s) { return bars + 8u * s; };
    auto bar_empty = [&](int s) { return bars + 8u * (STAGES + s); };
    const uint32_t verdict = bars + 16u * STAGES;  // one word: who finishes a cut tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), Cfg::CONSUMERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (tid == 32) {
        // the two descriptors travel while the barriers are being set up
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    }
    __syncthreads();
    launch_begin();  // nothing above touches global memory

    int64_t it_begin = (int64_t)blockIdx.x * g.iters_per_cta;
    int64_t it_end = min(g.total_iters, it_begin + g.iters_per_cta);
    const int pieces = g.pieces, piece = pieces > 1 ? (int)(blockIdx.x % (unsigned)pieces) : 0;
    if (pieces > 1) {
        // the CTAs of a tile share its k-iterations evenly
        const int64_t tile_first = (int64_t)(blockIdx.x / (unsigned)pieces) * g.k_iters;
        it_begin = tile_first + g.k_iters * piece / pieces;
        it_end = tile_first + g.k_iters * (piece + 1) / pieces;
    }
    const bool a_mn = !g.a_kfast, b_mn = !g.b_kfast;

    // ---------------------------------------------------------------- loads
    // They run `kLead` k-iterations ahead.  Issuing iteration j needs the slot that iteration
    // j - STAGES used, i.e. every warp must have finished that one; with kLead = STAGES - 2 that is
    // two iterations behind the issuing warp itself, so the wait is short.  The warps take turns, one
    // iteration each: a warp that issued them all was a third of an iteration behind the others
    // each time, and the whole CTA ran at its pace (chi = 512 chain, per product: 70.4 -> 68.0 us; f64 4000^3 3.99 ->
    // 3.90 ms; 300 x 300 x 4000 50 -> 39 us).
    constexpr int kLead = STAGES - 2;
    const uint32_t my_iters = (uint32_t)(it_end - it_begin);  // the host keeps total_iters below 2^31
    auto issue = [&](uint32_t j) {
        const uint32_t k_iters = (uint32_t)g.k_iters, tiles_m = (uint32_t)g.tiles_m, tiles_n = (uint32_t)g.tiles_n;
        const uint32_t at = (uint32_t)it_begin + j, tile = at / k_iters, rest = tile / tiles_m, bb = rest / tiles_n;
        const int m0 = (int)((tile - rest * tiles_m) * BM), n0 = (int)((rest - bb * tiles_n) * BN);
        const int k0 = (int)((at - tile * k_iters) * BK);
        const int s = (int)(j % STAGES);
        mbar_wait(bar_empty(s), ((j / STAGES) & 1) ^ 1, status, 0x301);
        const uint32_t a_dst = ring + s * Cfg::STAGE_BYTES, b_dst = a_dst + Cfg::A_BYTES;
        mbar_expect_tx(bar_full(s), Cfg::STAGE_BYTES);
        auto load = [&](const CUtensorMap* map, uint32_t dst, bool mn, bool runs, int r0, int rows) {
            if (!Cfg::kLines || !runs) {
                if (mn) tma_load_4d(dst, map, bar_full(s), 0, k0, r0 / Cfg::G, (int)bb);
                else    tma_load_4d(dst, map, bar_full(s), 0, r0, k0 / Cfg::KR, (int)bb);
            } else if (mn) {
                for (int r = 0; r < rows; r += Cfg::G)
                    tma_load_4d(dst + r * BK * ES, map, bar_full(s), 2 * (r0 + r), k0, 0, (int)bb);
            } else {
                for (int k = 0; k < BK; k += Cfg::KR)
                    tma_load_4d(dst + k * rows * ES, map, bar_full(s), 2 * (k0 + k), r0, 0, (int)bb);
            }
        };
        load(&map_a, a_dst, a_mn, g.a_runs, m0, BM);
        load(&map_b, b_dst, b_mn, g.b_runs, n0, BN);
    };
    // the first kLead iterations: one each, too
    for (uint32_t j = warp; lane == 0 && j < kLead && j < my_iters; j += Cfg::CONSUMERS) issue(j);

    // -------------------------------------------------------------------- consumers
    const int wm0 = (warp % Cfg::WARPS_M) * Cfg::WM, wn0 = (warp / Cfg::WARPS_M) * Cfg::WN;
    const int lr = lane >> 2, lc = lane & 3;
    const bool conj_a = g.conj_a != 0, conj_b = g.conj_b != 0;
    uint32_t n = 0;
    int64_t it = it_begin;
    while (it < it_end) {
        const int64_t tile = it / g.k_iters;
        const int64_t kb = it - tile * g.k_iters;
        const int64_t ke = min(g.k_iters, kb + (it_end - it));
        const int64_t tm = tile % g.tiles_m, rest = tile / g.tiles_m, tn = rest % g.tiles_n, bb = rest / g.tiles_n;
        const int64_t m0 = tm * BM, n0 = tn * BN;
        double acc[TM][TN][Cfg::ACC];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int e = 0; e < Cfg::ACC; ++e) acc[i][j][e] = 0.0;

        for (int64_t kit = kb; kit < ke; ++kit, ++n) {
            const int s = n % STAGES;
            if (lane == 0 && n % Cfg::CONSUMERS == (uint32_t)warp && n + kLead < my_iters) issue(n + kLead);
            if (lane == 0) mbar_wait(bar_full(s), (n / STAGES) & 1, status, 0x302);
            __syncwarp();
            const char* sa = smem + (size_t)s * Cfg::STAGE_BYTES;
            const char* sb = sa + Cfg::A_BYTES;
            if (a_mn) {
                if (b_mn) dmma_tma_consume<Cfg, true, true>(sa, sb, acc, wm0, wn0, lr, lc, conj_a, conj_b);
                else      dmma_tma_consume<Cfg, true, false>(sa, sb, acc, wm0, wn0, lr, lc, conj_a, conj_b);
            } else {
                if (b_mn) dmma_tma_consume<Cfg, false, true>(sa, sb, acc, wm0, wn0, lr, lc, conj_a, conj_b);
                else      dmma_tma_consume<Cfg, false, false>(sa, sb, acc, wm0, wn0, lr, lc, conj_a, conj_b);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty(s));
        }

        if constexpr (CPLX && !Cfg::kFour) {
            // fold the three products of this k range into Re (slots 0-1) and Im (slots 2-3)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double p1 = acc[i][j][e], p2 = conj_a != conj_b ? -acc[i][j][2 + e] : acc[i][j][2 + e], p3 = acc[i][j][4 + e];
                        acc[i][j][e] = p1 - p2;
                        acc[i][j][2 + e] = p3 - p1 - p2;
                    }
        }
        if (g.cluster > 1) {
            // The tile's sums meet in the CTAs' shared memory: each parks its own (the ring is empty: every load
            // that this CTA issued has been consumed), and adds a share of the tile over all of them, in the order
            // of k.
            __syncthreads();
            dmma_tma_park<Cfg>(smem, acc, tid);
            cluster_sync_all();
            constexpr int TOTAL = BM * BN;
            const int share = (TOTAL + pieces - 1) / pieces, at1 = min(TOTAL, (piece + 1) * share);
            for (int at = piece * share + tid; at < at1; at += Cfg::NT) {
                double xr = 0.0, xi = 0.0;
                const uint32_t mine = ring + (uint32_t)at * ES;
#pragma unroll 8
                for (int c = 0; c < pieces; ++c) {
                    const uint32_t q = map_to_cta(mine, (uint32_t)c);
                    if constexpr (CPLX) {
                        const double2 v = cluster_load_d2(q);
                        xr += v.x;
                        xi += v.y;
                    } else {
                        xr += cluster_load_d(q);
                    }
                }
                dmma_tma_store_one<Cfg>(g, bb, m0, n0, at / Cfg::NT, at % Cfg::NT, xr, xi);
            }
            __syncwarp();
            cluster_sync_all();  // no CTA leaves while another reads its sums
            break;
        }
        // A range that cuts a tile without a cluster: every CTA but one parks its sums in a scratch slot and counts
        // itself in; whoever comes last adds the slots in the order of k and writes C.  No CTA waits for another, so
        // nothing depends on which of them run at the same time.  Contributions (kb > 0) are the first thing a
        // CTA does and a tile's first range the last, so the range that starts the tile mostly finds the others
        // there and keeps its own sums in registers.
        bool finish = true;
        if (g.sk_two_phase) {
            dmma_tma_park<Cfg>(dmma_tma_slot<Cfg>(g, 0, blockIdx.x), acc, tid);
            finish = false;
        } else if (kb > 0 || ke < g.k_iters) {
            const int64_t first = tile * g.k_iters / g.iters_per_cta, last = ((tile + 1) * g.k_iters - 1) / g.iters_per_cta;
            const unsigned others = (unsigned)(last - first);
            unsigned* arrived = g.sk_arrived + first;
            auto told = [&]() -> bool {  // what thread 0 has put into the word
                __syncthreads();
                uint32_t v;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(verdict) : "memory");
                return v != 0;
            };
            auto count_in = [&]() -> bool {
                __threadfence();
                __syncthreads();
                if (tid == 0) {
                    unsigned before;
                    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(arrived) : "memory");
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(verdict), "r"((uint32_t)(before == others)) : "memory");
                }
                return told();
            };
            if (kb > 0) {
                dmma_tma_park<Cfg>(dmma_tma_slot<Cfg>(g, 0, blockIdx.x), acc, tid);
                finish = count_in();
                if (finish) {
                    __threadfence();
                    dmma_tma_gather<Cfg, false>(dmma_tma_slot<Cfg>(g, 1, first), acc, tid);
                }
            } else {
                __syncthreads();  // (the word may still be being read for the tile before)
                if (tid == 0) {
                    unsigned now;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(arrived) : "memory");
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(verdict), "r"((uint32_t)(now == others)) : "memory");
                }
                if (!told()) {
                    dmma_tma_park<Cfg>(dmma_tma_slot<Cfg>(g, 1, blockIdx.x), acc, tid);
                    finish = count_in();
                }
                __threadfence();
            }
            if (finish) {
                if (tid == 0) *arrived = 0;  // every range of the tile is in: the next launch counts from zero
#pragma unroll 2
                for (int64_t c = first + 1; c <= last; ++c) dmma_tma_gather<Cfg, true>(dmma_tma_slot<Cfg>(g, 0, c), acc, tid);
            }
        }
        if (finish) {
            const int64_t row0 = m0 + wm0 + lr, col0 = n0 + wn0 + 2 * lc;
            if (g.mul) apply_mul_fragments<CPLX>(g, bb, row0, col0, acc);
            char* Cb = g.c + g.off_c_b(bb) * (int64_t)ES;
            const bool read_c = g.beta_re != 0.0 || g.beta_im != 0.0;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t nn = col0 + 8 * j + e;
                    if (nn >= g.N) continue;
                    const int64_t cn = g.off_c_n(nn);
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        const int64_t m = row0 + 8 * i;
                        if (m >= g.M) continue;
                        dmma_store<CPLX>(g, Cb + (g.off_c_m(m) + cn) * (int64_t)ES, read_c, acc[i][j][e], acc[i][j][CPLX ? 2 + e : e]);
                    }
                }
            }
        }
        it += ke - kb;
    }
}

// Second phase of the two-launch split over K (outputs of a few tiles with a long K, such as
// 'abc,bcd->ad' with 64 x 64 outputs and K = 4096): every CTA of the main kernel has parked the
// sums of its k range in its slot; here one block per (tile, fragment) adds the `pieces` slots of
// a tile - one value per piece and thread, all loads independent, always in piece order, so the
// result does not depend on timing - and applies multiplier, alpha and beta.  The thread-to-element
// map is the main kernel's.  No CTA ever waits for another one.
template <typename Cfg>
__global__ void __launch_bounds__(Cfg::NT) dmma_tma_splitk_finish_kernel(ContractArgs g, int pieces) {
    constexpr bool CPLX = Cfg::kCplx;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, ES = Cfg::ES;
    launch_begin();
    const int64_t tile = blockIdx.x;
    const int f = blockIdx.y, tid = threadIdx.x;
    const int64_t tm = tile % g.tiles_m, rest = tile / g.tiles_m, tn = rest % g.tiles_n, bb = rest / g.tiles_n;
    const char* P = g.partial + ((size_t)tile * pieces * (BM * BN) + (size_t)f * Cfg::NT + tid) * ES;
    double xr = 0.0, xi = 0.0;
#pragma unroll 8
    for (int s = 0; s < pieces; ++s) {
        const char* q = P + (size_t)s * (BM * BN) * ES;
        if (CPLX) {
            const double2 v = __ldcg(reinterpret_cast<const double2*>(q));
            xr += v.x;
            xi += v.y;
        } else {
            xr += __ldcg(reinterpret_cast<const double*>(q));
        }
    }
    dmma_tma_store_one<Cfg>(g, bb, tm * BM, tn * BN, f, tid, xr, xi);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledF64)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledF64 encode_tiled_f64() {
    static EncodeTiledF64 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiledF64)p;
    }();
    return fn;
}

// Tensor map of one operand (free group `fr`, tensor index tns); false when TMA cannot describe it.
// *runs: one load per run (see the top of this file).
template <typename Cfg>
static bool make_f64_map(const ContractProblem& p, const std::vector<Mode>& fr, int tns, const void* base, int rows,
                         bool* mn_major, bool* runs, CUtensorMap* map) {
    EncodeTiledF64 enc = encode_tiled_f64();
    F64MapShape d;
    if (!enc || !f64_map_shape(p, fr, tns, base, rows, F64MapForm{Cfg::kCplx, Cfg::kLines, Cfg::KR, Cfg::G, Cfg::BK}, &d)) return false;
    *mn_major = d.mn_major;
    *runs = d.runs;
    const cuuint64_t dims[4] = {d.dims[0], d.dims[1], d.dims[2], d.dims[3]}, strides[3] = {d.strides[0], d.strides[1], d.strides[2]};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(base), dims, strides, d.box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, Cfg::kLines ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTAs of a cluster that share a tile's K, 0 for none: where all those clusters run at once, which what a
// CTA takes of an SM decides (`fit`, by size: with 200 KB of shared memory 74 of two, 33 of four, 15 of eight), and no CTA
// has more k-iterations than one of the ranges below would, or one more of the short iterations of the small tiles (half a
// microsecond).  The sums then meet in shared memory, half a microsecond to two earlier than through scratch and counters
// (us by cluster, by ranges: double, 56 tiles of 32 x 32 and K = 256 in two 9.8, 11.4, 18 and K = 1024 in eight 9.6, 11.6; complex,
// 97 x 194 x 97 9.5, 10.7, 64 x 128 x 64 8.0, 9.8; in two turns, 36 tiles in four, 23.2, 13.8; 512 x 512 x 1024, 16 iterations
// of 64 x 64 tiles against 14, 70.2, 67.5).
template <typename Cfg>
static int cluster_pieces(const ContractArgs& a, int64_t slots, const int (&fit)[3]) {
    if (!env_int("TFB_DMMA_CLUSTER", 1)) return 0;
    const int64_t ranges = std::min<int64_t>(slots, std::max<int64_t>(1, a.total_iters / 2));
    const int64_t most = (a.total_iters + ranges - 1) / ranges + (Cfg::BM * Cfg::BN * Cfg::BK * (Cfg::kCplx ? 3 : 1) <= 65536);
    for (int i = 2; i >= 0; --i) {
        const int s = 2 << i;
        if (a.k_iters >= s && a.n_tiles <= fit[i] && a.n_tiles * s <= slots && (a.k_iters + s - 1) / s <= most) return s;
    }
    return 0;
}
template <typename Cfg>
static tfb_status clusters_that_fit(int (&fit)[3]) {
    for (int i = 0; i < 3; ++i) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2u << i;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(2u << i);
        cfg.blockDim = dim3(Cfg::NT);
        cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        TFB_CUDA(cudaOccupancyMaxActiveClusters(&fit[i], contract_dmma_tma_kernel<Cfg>, &cfg));
    }
    return TFB_OK;
}

// Runs the TMA-fed kernel when both operands qualify; otherwise *declined = true.
template <typename Cfg>
static tfb_status run_tma_cfg(tfb_ctx* ctx, const ContractProblem& p, ContractArgs a, bool* declined) {
    using Base = typename Cfg::Base;
    *declined = true;
    if (a.M > INT32_MAX - 512 || a.N > INT32_MAX - 512 || a.K > INT32_MAX - 64) return TFB_OK;
    CUtensorMap map_a, map_b;
    bool a_mn = false, b_mn = false, a_runs = false, b_runs = false;
    if (!make_f64_map<Cfg>(p, p.m, 0, p.a, Cfg::BM, &a_mn, &a_runs, &map_a)) return TFB_OK;
    if (!make_f64_map<Cfg>(p, p.n, 1, p.b, Cfg::BN, &b_mn, &b_runs, &map_b)) return TFB_OK;
    a.a_kfast = !a_mn;
    a.b_kfast = !b_mn;
    a.a_runs = a_runs;
    a.b_runs = b_runs;
    static std::mutex mu;
    struct Fit { int clusters[3]; };
    static std::map<int, Fit> configured;
    Fit fit;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = configured.find(ctx->device);
        if (it == configured.end()) {
            TFB_CUDA(cudaFuncSetAttribute(contract_dmma_tma_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          Cfg::SMEM_BYTES));
            TFB_TRY(clusters_that_fit<Cfg>(fit.clusters));
            it = configured.emplace(ctx->device, fit).first;
        }
        fit = it->second;
    }
    a.tiles_m = (a.M + Cfg::BM - 1) / Cfg::BM;
    a.tiles_n = (a.N + Cfg::BN - 1) / Cfg::BN;
    a.n_tiles = a.tiles_m * a.tiles_n * a.B;
    a.k_iters = (a.K + Cfg::BK - 1) / Cfg::BK;
    a.total_iters = a.n_tiles * a.k_iters;
    if (a.total_iters >= ((int64_t)1 << 31)) return TFB_OK;  // the producer indexes k-iterations with 32 bits
    const int64_t slots = ctx->sm_count;  // one CTA per SM
    int64_t grid = 0;
    int pieces = 0;
    a.cluster = cluster_pieces<Cfg>(a, slots, fit.clusters);
    if (a.cluster > 1) grid = a.n_tiles * a.cluster;
    // A handful of tiles with a long K: cut every tile into the same number of k pieces, as even as its iterations allow, one CTA
    // each, and add the pieces in a second, tiny launch.  (In one launch the
    // last range of a tile adds all its pieces - dependent round trips to L2 - and 'abc,bcd->ad' at 64^4 took 16.4 us; here every
    // load of the sum is independent.  us in one launch and so: double, 24 x 1044 x 992 20.5, 17.6, 128 x 128 x 5000 26.6, 19.6, 156 x
    // 80 x 6752 31.3, 24.5; complex 16 x 12 x 5128 24.6, 20.5.)
    if (!grid && a.n_tiles * 4 <= slots && a.k_iters * Cfg::BK >= 256 && env_int("TFB_SK_TWO_PHASE", 1)) {
        const int64_t want = std::min<int64_t>(std::min<int64_t>(32, slots / a.n_tiles), a.k_iters * Cfg::BK / 64);
        // (32-deep iterations do not deal out as evenly: where the longest piece is longer than the equal ranges below, those are
        // ahead: 344 x 312 x 280 complex double in 90 pieces of three iterations 23.8 us, 19.9)
        if (want >= 2 && (Cfg::BK <= 16 || (a.k_iters + want - 1) / want <= (a.total_iters + slots - 1) / slots)) pieces = (int)want;
        if (pieces) {
            grid = a.n_tiles * pieces;
            a.sk_two_phase = 1;
        }
    }
    if (!grid) {
        if (a.n_tiles % slots == 0 || a.n_tiles >= 16 * slots) {
            grid = std::min(a.n_tiles, slots);
            a.iters_per_cta = ((a.n_tiles + grid - 1) / grid) * a.k_iters;
        } else {
            // At least two k-iterations per CTA (eight launches of a chain, chi = 64: 98 -> 84 us against
            // at least four).
            grid = std::min<int64_t>(slots, std::max<int64_t>(1, a.total_iters / 2));
            a.iters_per_cta = (a.total_iters + grid - 1) / grid;
            // Whoever finishes a tile passes over a slot per range of it: keep a tile in at most 32.
            a.iters_per_cta = std::max<int64_t>(a.iters_per_cta, (a.k_iters + 31) / 32);
        }
        grid = (a.total_iters + a.iters_per_cta - 1) / a.iters_per_cta;
    }
    a.pieces = a.cluster > 1 ? a.cluster : pieces;
    if (a.sk_two_phase || (a.cluster <= 1 && a.iters_per_cta % a.k_iters != 0)) {
        // Scratch slots and counters live with the context and are reused by every launch (a counter is back at zero
        // when its tile is finished, so a replayed launch finds what a direct one does).
        // As large as any configuration asks for from the start (38 MB): a captured launch keeps the address.  Where the
        // device has no room for that, what this launch uses.
        static_assert((size_t)Base::TILE_ELEMS * Base::ES <= 128 * 128 * 8, "largest block tile");
        if ((size_t)grid > tfb_ctx::kArrived) return fail(TFB_ERR_DEVICE, "a device of more than %zu SMs", tfb_ctx::kArrived);
        const size_t need = (a.sk_two_phase ? 1 : 2) * (size_t)grid * Base::TILE_ELEMS * Base::ES;
        if (ctx->sk_partial_bytes < need) {
            if (ctx->sk_partial) TFB_CUDA(cudaFree(ctx->sk_partial));
            ctx->sk_partial = nullptr;
            ctx->sk_partial_bytes = 0;
            size_t take = 2 * std::max<size_t>((size_t)grid, (size_t)slots) * 128 * 128 * 8;
            if (cudaMalloc(&ctx->sk_partial, take) != cudaSuccess) {
                cudaGetLastError();
                take = need;
                TFB_CUDA(cudaMalloc(&ctx->sk_partial, take));
            }
            ctx->sk_partial_bytes = take;
        }
        a.partial = (char*)ctx->sk_partial;
        a.sk_arrived = ctx->arrived;
    }
    {
        LaunchScope ls(ctx, "contract_dmma");
        int* status = ctx->dev_status;
        TFB_CUDA(launch_overlapped(ctx, contract_dmma_tma_kernel<Cfg>, dim3((unsigned)grid), dim3(Cfg::NT), Cfg::SMEM_BYTES,
                                   (unsigned)a.cluster, map_a, map_b, a, status));
    }
    if (a.sk_two_phase) {
        LaunchScope ls(ctx, "contract_dmma_finish");
        TFB_CUDA(launch_overlapped(ctx, dmma_tma_splitk_finish_kernel<Cfg>, dim3((unsigned)a.n_tiles, Cfg::TM * Cfg::TN * 2),
                                   dim3(Cfg::NT), 0, 0u, a, pieces));
    }
    *declined = false;
    return TFB_OK;
}

}  // namespace tfb
