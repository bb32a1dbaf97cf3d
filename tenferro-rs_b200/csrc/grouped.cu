// Grouped (ragged) matrix products in one persistent launch.  `PrimDescriptor::BatchedGemm`
// (tenferro-prims/src/lib.rs:156-168) covers uniform batches; a table of problems with
// individual sizes carries the same C = alpha * A * B + beta * C to ragged batches such as the
// sector blocks of a block-sparse tensor pair.
//
// This file holds the kernel for every table the f32 tensor-core kernels decline - double
// precision, complex, f32 of any size, alignment and strides - and the entry points.
//
// Such a table is bound by latency: a block of 40 x 40 x 40 doubles is 38 KB and 0.5 us of one SM's
// FP64 pipe.  So the kernel is arranged to wait for memory once and not per problem:
//   * a unit of work is one output tile (64 x 64 real, 32 x 32 complex); the host deals
//     them out when the table is prepared, longest first, each to the CTA with the least work so
//     far, so nothing is uploaded, sorted or drawn from a ticket per call;
//   * a CTA walks its list in 32-deep k stages through a ring of cp.async stages that runs across
//     units: while one unit is computed and stored the next ones' operands are on their way;
//   * f64 and Complex64 run on the FP64 tensor pipe (m16n8k8; four real products per complex one, so
//     that Re and Im each keep their own accuracy), f32 and Complex32 as FMAs (exact products);
//   * the four warps tile a unit as 2 x 2, 4 x 1 or 1 x 4 fragment blocks, whichever leaves the
//     least padding, and dead blocks are not issued.
// Measured against one thread-per-output tile drawn from an atomic ticket, the table uploaded per call:
// 1024 f64 blocks with sides 4 .. 160 (41 MB, 128 MFLOP, floor 6 us of HBM) 159 -> 25.6 us a run, 4096 of
// them 82 us, f32 with such sides 183 -> 25 us.  What a table runs out of is issue slots and, while it is small, the longest
// block's chain of stages: 32-deep stages, two of them, instead of 16-deep ones, three (64 blocks 16.5 -> 14.4 us, 1024 26.7 -> 25.6,
// f32 28.4 -> 24.7), fetches worked out once a unit (64: 18.5 -> 16.5; 1024 with sides 16 .. 128 34.4 -> 31.2) and
// one addition per stored element (1024: 30.9 -> 26.2, 4096: 101 -> 84).  Eight warps a CTA double the units' fixed instructions
// (1024: 55.6 us).
#include "common.h"
#include "contract_common.cuh"
#include "grouped_layout.h"
#include "scalar_ops.cuh"

namespace tfb {

namespace {

constexpr int kGroupThreads = 128;

template <typename T>
struct GroupSmem {
    using Cfg = GroupCfg<T>;
    static constexpr int KFAST = Cfg::TILE * Cfg::PK, MFAST = kGroupK * Cfg::PM;
    static constexpr int ELEMS = KFAST > MFAST ? KFAST : MFAST;  // of one operand
    static constexpr int STAGE = 2 * ELEMS * (int)sizeof(T);
    static constexpr int RECS = kGroupRecs * (int)sizeof(GroupUnit);
    static constexpr int BYTES = RECS + Cfg::STAGES * STAGE;
};

struct GroupedArgs {
    const GroupUnit* units;  // CTA c owns units[starts[c]] .. units[starts[c + 1])
    const int* starts;
    double alpha_re, alpha_im, beta_re, beta_im;
};

__device__ __forceinline__ void cp_async_part(uint32_t dst, const void* src, int bytes16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes16));
}
template <int ES>
__device__ __forceinline__ void cp_async_one(uint32_t dst, const void* src, int bytes) {
    if constexpr (ES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
    else if constexpr (ES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

// How this thread fetches its part of one operand's stages, worked out once per unit: what is left per stage is the copies and
// the additions between them.  (Worked out for every stage, the strides read anew, it was most of a stage's 480 instructions a warp
// where units are small, and issue slots are what such a table runs out of: ncu, 1024 f64 blocks, 37 % of them in use at 2.8 warps a
// scheduler, 10 % of DRAM.)
// A stage is up to 32 of K; what lies past a live k is filled with zeros up to the next multiple of 8, which is
// as far as the arithmetic reads; rows past the live ones may hold anything, nothing stored
// depends on them (V > 1: a chunk's dead part is zero-filled).
template <typename T>
struct OperandFeed {
    using Cfg = GroupCfg<T>;
    static constexpr int ES = (int)sizeof(T), VEC = 16 / ES;
    const T* p;        // this thread's first element of the next stage
    const T* corner;   // a valid address for copies of nothing
    int64_t step, adv; // elements from one of its copies to the next, from a stage to the next
    uint32_t off;      // of the first one inside the operand's part of a stage
    int dstep;         // bytes between them
    int n;             // k fast: copies of a stage.  Row fast: 0 or 1, whether it has any
    int k, kstep;      // k of the first copy, from one to the next (row fast)
    int live;          // bytes of a copy (row fast)
    bool kfast, vec;

    // `rows` rows with row stride rs, k with stride ks.
    __device__ __forceinline__ void set(const T* src, int64_t rs, int64_t ks, int rows, bool is_kfast, bool is_vec, int tid) {
        const int V = VEC > 1 && is_vec ? VEC : 1;
        corner = src;
        kfast = is_kfast;
        vec = is_vec;
        adv = kGroupK * ks;
        int r;
        if (kfast) {
            const int kc = kGroupK / V, per = kGroupThreads / kc;
            r = tid / kc;
            k = (tid - r * kc) * V;
            n = r < rows ? (rows - r + per - 1) / per : 0;
            step = per * rs;
            off = (uint32_t)((r * Cfg::PK + k) * ES);
            dstep = per * Cfg::PK * ES;
        } else {
            // a power-of-two group of threads along the rows
            const int chunks = (rows + V - 1) / V;
            int lg = 2;
            while ((1 << lg) < chunks) ++lg;
            const int x = tid & ((1 << lg) - 1);
            r = x * V;
            k = tid >> lg;
            kstep = kGroupThreads >> lg;
            n = x < chunks;
            live = min(rows - r, V) * ES;
            step = kstep * ks;
            off = (uint32_t)((k * Cfg::PM + r) * ES);
            dstep = kstep * Cfg::PM * ES;
        }
        p = src + r * rs + k * ks;
    }
    template <int V>
    __device__ __forceinline__ void copies(uint32_t d, int kv) {
        const int kr = (kv + 7) & ~7;
        auto copy = [&](const T* q, int bytes) {
            if constexpr (V == 1) cp_async_one<ES>(d, q, bytes);
            else cp_async_part(d, q, bytes);
            d += dstep;
        };
        if (kfast) {
            if (k >= kr) return;
            const int bytes = min(max(kv - k, 0), V) * ES;
            const T* q = bytes ? p : corner;
            const int64_t s = bytes ? step : 0;
#pragma unroll 4
            for (int i = 0; i < n; ++i, q += s) copy(q, bytes);
        } else if (n) {
            const T* q = p;
#pragma unroll 4
            for (int kk = k; kk < kr; kk += kstep, q += step) copy(kk < kv ? q : corner, kk < kv ? live : 0);
        }
    }
    // The next stage, `kv` <= 32 of K live.
    __device__ __forceinline__ void stage(uint32_t dst, int kv) {
        if (VEC > 1 && vec) copies<VEC>(dst + off, kv);
        else copies<1>(dst + off, kv);
        p += adv;
    }
};

__device__ __forceinline__ void group_dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Runs CALL(NI, NJ) with the live block counts as compile-time constants: a small unit then issues
// only its own instructions.
#define TFB_GROUP_CASE(I, J, CALL) \
    if constexpr ((I) <= Cfg::NI && (J) <= Cfg::NJ) { if (ni == (I) && nj == (J)) { CALL(I, J); return; } }

// The FP64 tensor pipe.  Fragment numbering of m16n8k8: A rows g and g + 8, k = t and t + 4; C columns 2t, 2t + 1.
template <typename T>
struct TensorPath {
    using Cfg = GroupCfg<T>;
    static constexpr bool CPLX = Ops<T>::is_complex;
    static constexpr int W = CPLX ? 2 : 1;
    double acc[Cfg::NI][Cfg::NJ][W][4];
    int wm, wn, ni, nj;

    __device__ __forceinline__ void begin(const GroupUnit& u, int tid) {
        const int warp = tid >> 5;
        const int lw = u.shape & 3, pi = (u.shape >> 2) & 3, pj = (u.shape >> 4) & 15;
        wm = (warp & ((1 << lw) - 1)) * 16 * pi;
        wn = (warp >> lw) * 8 * pj;
        ni = max(0, min(pi, ((int)u.mt - wm + 15) / 16));
        nj = max(0, min(pj, ((int)u.nt - wn + 7) / 8));
#pragma unroll
        for (int i = 0; i < Cfg::NI; ++i)
#pragma unroll
            for (int j = 0; j < Cfg::NJ; ++j)
#pragma unroll
                for (int w = 0; w < W; ++w)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][j][w][e] = 0.0;
    }
    template <int NI, int NJ>
    __device__ __forceinline__ void stage_t(const T* As, const T* Bs, int a_sm, int a_sk, int b_sn, int b_sk, int steps, int tid) {
        const int g = (tid & 31) >> 2, t = tid & 3;
        const T* pa = As + (wm + g) * a_sm + t * a_sk;
        const T* pb = Bs + (wn + g) * b_sn + t * b_sk;
        for (int s = 0; s < steps; ++s, pa += 8 * a_sk, pb += 8 * b_sk) {
            T av[NI][4], bv[NJ][2];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) av[i][e] = pa[(16 * i + 8 * (e & 1)) * a_sm + 4 * (e >> 1) * a_sk];
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) bv[j][e] = pb[8 * j * b_sn + 4 * e * b_sk];
            if constexpr (CPLX) {
                double ar[NI][4], ai[NI][4], an[NI][4], br[NJ][2], bi[NJ][2];
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) { ar[i][e] = av[i][e].x; ai[i][e] = av[i][e].y; an[i][e] = -av[i][e].y; }
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) { br[j][e] = bv[j][e].x; bi[j][e] = bv[j][e].y; }
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) { group_dmma(acc[i][j][0], ar[i], br[j]); group_dmma(acc[i][j][1], ar[i], bi[j]); }
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) { group_dmma(acc[i][j][0], an[i], bi[j]); group_dmma(acc[i][j][1], ai[i], br[j]); }
            } else {
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) group_dmma(acc[i][j][0], av[i], bv[j]);
            }
        }
    }
    __device__ __forceinline__ void stage(const T* As, const T* Bs, int a_sm, int a_sk, int b_sn, int b_sk, int kv, int tid) {
        const int steps = (kv + 7) >> 3;
#define TFB_CALL(I, J) stage_t<I, J>(As, Bs, a_sm, a_sk, b_sn, b_sk, steps, tid)
        TFB_GROUP_CASE(1, 1, TFB_CALL) TFB_GROUP_CASE(1, 2, TFB_CALL) TFB_GROUP_CASE(1, 3, TFB_CALL) TFB_GROUP_CASE(1, 4, TFB_CALL)
        TFB_GROUP_CASE(2, 1, TFB_CALL) TFB_GROUP_CASE(2, 2, TFB_CALL) TFB_GROUP_CASE(2, 3, TFB_CALL) TFB_GROUP_CASE(2, 4, TFB_CALL)
#undef TFB_CALL
    }
    __device__ __forceinline__ void store(const GroupUnit& u, T alpha, T beta, bool read_c, int tid) {
        const int g = (tid & 31) >> 2, t = tid & 3;
        // a thread's rows are eight apart, its columns two neighbours of every eight: one addition an element
        const int m0 = wm + g, n0 = wn + 2 * t, rows = ((int)u.mt - m0 + 7) >> 3;
        const int64_t row8 = 8 * u.c_rs, cs = u.c_cs;
        T* col = reinterpret_cast<T*>(u.c) + m0 * u.c_rs + n0 * cs;
#pragma unroll
        for (int j = 0; j < Cfg::NJ; ++j) {
            if (j < nj) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (n0 + 8 * j + e < u.nt) {
                        T* p = col + e * cs;
#pragma unroll
                        for (int r = 0; r < 2 * Cfg::NI; ++r, p += row8) {
                            if (r < 2 * ni && r < rows) {
                                T x;
                                if constexpr (CPLX) x = make_double2(acc[r >> 1][j][0][2 * (r & 1) + e], acc[r >> 1][j][1][2 * (r & 1) + e]);
                                else x = acc[r >> 1][j][0][2 * (r & 1) + e];
                                T v = Ops<T>::mul(alpha, x);
                                if (read_c) v = Ops<T>::add(v, Ops<T>::mul(beta, *p));
                                *p = v;
                            }
                        }
                    }
                }
                col += 8 * cs;
            }
        }
    }
};

// FMAs: 16 x 8 threads, rows tx + 16 i, columns ty + 8 j.
template <typename T>
struct FmaPath {
    using Cfg = GroupCfg<T>;
    T acc[Cfg::NI][Cfg::NJ];
    int ni, nj;

    __device__ __forceinline__ void begin(const GroupUnit& u, int) {
        // block counts rounded up to powers of two: nine forms instead of thirty-two
        ni = u.mt <= 16 ? 1 : u.mt <= 32 ? 2 : 4;
        nj = u.nt <= 8 ? 1 : u.nt <= 16 ? 2 : u.nt <= 32 ? 4 : 8;
#pragma unroll
        for (int i = 0; i < Cfg::NI; ++i)
#pragma unroll
            for (int j = 0; j < Cfg::NJ; ++j) acc[i][j] = Ops<T>::zero();
    }
    template <int NI, int NJ>
    __device__ __forceinline__ void stage_t(const T* As, const T* Bs, int a_sm, int a_sk, int b_sn, int b_sk, int kr, int tid) {
        const T* pa = As + (tid & 15) * a_sm;
        const T* pb = Bs + (tid >> 4) * b_sn;
#pragma unroll 4
        for (int k = 0; k < kr; ++k, pa += a_sk, pb += b_sk) {
            T av[NI], bv[NJ];
#pragma unroll
            for (int i = 0; i < NI; ++i) av[i] = pa[16 * i * a_sm];
#pragma unroll
            for (int j = 0; j < NJ; ++j) bv[j] = pb[8 * j * b_sn];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[i][j] = Ops<T>::fma_(av[i], bv[j], acc[i][j]);
        }
    }
    __device__ __forceinline__ void stage(const T* As, const T* Bs, int a_sm, int a_sk, int b_sn, int b_sk, int kv, int tid) {
        const int kr = (kv + 3) & ~3;
#define TFB_CALL(I, J) stage_t<I, J>(As, Bs, a_sm, a_sk, b_sn, b_sk, kr, tid)
        TFB_GROUP_CASE(1, 1, TFB_CALL) TFB_GROUP_CASE(1, 2, TFB_CALL) TFB_GROUP_CASE(1, 4, TFB_CALL) TFB_GROUP_CASE(1, 8, TFB_CALL)
        TFB_GROUP_CASE(2, 1, TFB_CALL) TFB_GROUP_CASE(2, 2, TFB_CALL) TFB_GROUP_CASE(2, 4, TFB_CALL) TFB_GROUP_CASE(2, 8, TFB_CALL)
        TFB_GROUP_CASE(4, 1, TFB_CALL) TFB_GROUP_CASE(4, 2, TFB_CALL) TFB_GROUP_CASE(4, 4, TFB_CALL) TFB_GROUP_CASE(4, 8, TFB_CALL)
#undef TFB_CALL
    }
    __device__ __forceinline__ void store(const GroupUnit& u, T alpha, T beta, bool read_c, int tid) {
        const int tx = tid & 15, ty = tid >> 4, rows = ((int)u.mt - tx + 15) >> 4;
        const int64_t row16 = 16 * u.c_rs, col8 = 8 * u.c_cs;
        T* col = reinterpret_cast<T*>(u.c) + tx * u.c_rs + ty * u.c_cs;
#pragma unroll
        for (int j = 0; j < Cfg::NJ; ++j, col += col8) {
            if (ty + 8 * j < u.nt) {
                T* p = col;
#pragma unroll
                for (int i = 0; i < Cfg::NI; ++i, p += row16) {
                    if (i < rows) {
                        T v = Ops<T>::mul(alpha, acc[i][j]);
                        if (read_c) v = Ops<T>::add(v, Ops<T>::mul(beta, *p));
                        *p = v;
                    }
                }
            }
        }
    }
};
#undef TFB_GROUP_CASE

template <typename T, typename Path>
__global__ void __launch_bounds__(kGroupThreads, GroupCfg<T>::CTAS) grouped_units_kernel(GroupedArgs g) {
    using Cfg = GroupCfg<T>;
    using Sm = GroupSmem<T>;
    constexpr int S = Cfg::STAGES;
    extern __shared__ __align__(16) char group_smem[];
    const GroupUnit* recs = reinterpret_cast<const GroupUnit*>(group_smem);
    const uint32_t rec_addr = (uint32_t)__cvta_generic_to_shared(group_smem), ring_addr = rec_addr + Sm::RECS;
    const int tid = threadIdx.x;
    const int first = g.starts[blockIdx.x], n_units = g.starts[blockIdx.x + 1] - first;
    if (n_units <= 0) return;
    const char* table = reinterpret_cast<const char*>(g.units + first);
    for (int c = tid; c < min(n_units, kGroupRecs) * kGroupRecChunks; c += kGroupThreads)
        cp_async_part(rec_addr + 16 * c, table + 16 * c, 16);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();

    // The next stage to request: unit pu, `left` of its K.  At most S - 1 units ahead of the unit being
    // computed, so its record is in the shared window of kGroupRecs.
    int pu = 0, pk = 0;  // (pk: whether it has begun)
    int64_t left = 0;
    OperandFeed<T> feed_a, feed_b;
    auto request = [&](int slot) {
        if (pu < n_units) {
            if (pk == 0) {
                const GroupUnit& u = recs[pu % kGroupRecs];
                left = u.k;
                feed_a.set(reinterpret_cast<const T*>(u.a), u.a_rs, u.a_cs, u.mt, u.shape & kAFast, u.shape & kAVec, tid);
                feed_b.set(reinterpret_cast<const T*>(u.b), u.b_cs, u.b_rs, u.nt, u.shape & kBFast, u.shape & kBVec, tid);
            }
            const int kv = (int)min((int64_t)kGroupK, left);
            const uint32_t da = ring_addr + slot * Sm::STAGE, db = da + Sm::ELEMS * (int)sizeof(T);
            feed_a.stage(da, kv);
            feed_b.stage(db, kv);
            pk = 1;
            left -= kGroupK;
            if (left <= 0) {
                pk = 0;
                ++pu;
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < S - 1; ++s) request(s);

    const T alpha = Ops<T>::from(Scalar{g.alpha_re, g.alpha_im}), beta = Ops<T>::from(Scalar{g.beta_re, g.beta_im});
    const bool read_c = g.beta_re != 0 || g.beta_im != 0;
    Path path;
    int slot = 0, next_slot = S - 1;
    for (int cu = 0; cu < n_units; ++cu) {
        const GroupUnit& u = recs[cu % kGroupRecs];
        const int64_t K = u.k;
        const int a_sm = u.shape & kAFast ? Cfg::PK : 1, a_sk = u.shape & kAFast ? 1 : Cfg::PM;
        const int b_sn = u.shape & kBFast ? Cfg::PK : 1, b_sk = u.shape & kBFast ? 1 : Cfg::PM;
        path.begin(u, tid);
        int64_t k0 = 0;
        do {
            cp_async_wait<S - 2>();
            __syncthreads();
            if (k0 == 0 && cu > 0 && cu - 1 + kGroupRecs < n_units && tid < kGroupRecChunks)
                // every thread has left the unit before: its record makes room (lands with the stage below)
                cp_async_part(rec_addr + ((cu - 1) % kGroupRecs) * (int)sizeof(GroupUnit) + 16 * tid,
                              table + (int64_t)(cu - 1 + kGroupRecs) * sizeof(GroupUnit) + 16 * tid, 16);
            request(next_slot);
            __syncwarp();  // the requests' branches end here: the MMAs below need whole warps
            const T* As = reinterpret_cast<const T*>(group_smem + Sm::RECS + slot * Sm::STAGE);
            path.stage(As, As + Sm::ELEMS, a_sm, a_sk, b_sn, b_sk, (int)min((int64_t)kGroupK, K - k0), tid);
            if (++slot == S) slot = 0;
            if (++next_slot == S) next_slot = 0;
            k0 += kGroupK;
        } while (k0 < K);
        path.store(u, alpha, beta, read_c, tid);
    }
    cp_async_wait<0>();
}

// The CTAs' unit lists of one table, on the device.
struct GroupedUnits {
    PoolBlock mem;
    size_t starts_at = 0;
    int grid = 0;
};

tfb_status check_table(size_t n, const tfb_gemm_problem* problems) {
    for (size_t p = 0; p < n; ++p) {
        const auto& q = problems[p];
        if (q.m < 0 || q.n < 0 || q.k < 0) return fail(TFB_ERR_INVALID_ARGUMENT, "problem %zu has a negative size", p);
        if (q.m > 0 && q.n > 0 && (!q.c || (q.k > 0 && (!q.a || !q.b))))
            return fail(TFB_ERR_INVALID_ARGUMENT, "problem %zu has a NULL pointer", p);
    }
    return TFB_OK;
}

template <typename T>
tfb_status lay_out_units(tfb_ctx* ctx, size_t n, const tfb_gemm_problem* problems, bool balance, GroupedUnits* out) {
    static thread_local LayoutScratch scratch;
    size_t bytes = 0;
    TFB_TRY(deal_units<T>(n, problems, ctx->sm_count, balance, scratch, &bytes, &out->starts_at, &out->grid));
    if (out->grid == 0) return TFB_OK;
    TFB_TRY(out->mem.upload(ctx, scratch.table.data(), bytes));
    scratch.trim();
    return TFB_OK;
}

template <typename T, typename Path>
tfb_status launch_units(tfb_ctx* ctx, const GroupedUnits& f, Scalar alpha, Scalar beta, const char* name) {
    static std::mutex mu;
    static std::map<int, bool> configured;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[ctx->device]) {
            TFB_CUDA(cudaFuncSetAttribute(grouped_units_kernel<T, Path>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          GroupSmem<T>::BYTES));
            configured[ctx->device] = true;
        }
    }
    GroupedArgs g{(const GroupUnit*)f.mem.ptr, (const int*)((const char*)f.mem.ptr + f.starts_at), alpha.re, alpha.im, beta.re, beta.im};
    LaunchScope ls(ctx, name);
    grouped_units_kernel<T, Path><<<f.grid, kGroupThreads, GroupSmem<T>::BYTES, ctx->stream>>>(g);
    TFB_CUDA(cudaGetLastError());
    return TFB_OK;
}

tfb_status lay_out(tfb_ctx* ctx, int dtype, size_t n, const tfb_gemm_problem* problems, bool balance, GroupedUnits* out) {
    switch (dtype) {
        case TFB_F32: return lay_out_units<float>(ctx, n, problems, balance, out);
        case TFB_F64: return lay_out_units<double>(ctx, n, problems, balance, out);
        case TFB_C32: return lay_out_units<float2>(ctx, n, problems, balance, out);
        case TFB_C64: return lay_out_units<double2>(ctx, n, problems, balance, out);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

tfb_status run_units(tfb_ctx* ctx, int dtype, const GroupedUnits& f, Scalar alpha, Scalar beta) {
    if (f.grid == 0) return TFB_OK;
    switch (dtype) {
        case TFB_F32: return launch_units<float, FmaPath<float>>(ctx, f, alpha, beta, "grouped_simt");
        case TFB_F64: return launch_units<double, TensorPath<double>>(ctx, f, alpha, beta, "grouped_dmma");
        case TFB_C32: return launch_units<float2, FmaPath<float2>>(ctx, f, alpha, beta, "grouped_simt");
        case TFB_C64: return launch_units<double2, TensorPath<double2>>(ctx, f, alpha, beta, "grouped_dmma");
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

}  // namespace

}  // namespace tfb

// A problem table prepared once: the f32 tensor-core schedule on the device when the table
// qualifies, else the unit lists of the general kernel.
struct tfb_grouped_plan {
    tfb_ctx* ctx = nullptr;
    int dtype = 0;
    bool fast = false;
    tfb::GroupedFast schedule;
    tfb::GroupedUnits units;
    tfb_status invalid = TFB_OK;  // what is wrong with the table: reported by every execute
    std::string why;
};

namespace {

tfb_status prepare(tfb_ctx* ctx, int dtype, size_t n, const tfb_gemm_problem* problems, bool balance, tfb_grouped_plan* plan) {
    using namespace tfb;
    DeviceGuard g(ctx->device);
    plan->ctx = ctx;
    plan->dtype = dtype;
    if (dtype == TFB_F32) {
        // The mma.sync kernel is the faster one on the tables it takes (dims in multiples of 16, K up to
        // 128); the tcgen05 kernel takes any dims with 16-byte aligned columns and K up to 512; the
        // general kernel takes everything.
        const bool tcgen05_first = env_int("TFB_GROUPED_PREFER_TCGEN05", 0) != 0;
        bool declined = true;
        if (tcgen05_first) TFB_TRY(grouped_tcgen05_prepare(ctx, n, problems, &plan->schedule, &declined));
        if (declined) TFB_TRY(grouped_tf32_prepare(ctx, n, problems, &plan->schedule, &declined));
        if (declined && !tcgen05_first) TFB_TRY(grouped_tcgen05_prepare(ctx, n, problems, &plan->schedule, &declined));
        plan->fast = !declined;
    }
    if (plan->fast) return TFB_OK;
    plan->invalid = check_table(n, problems);
    if (plan->invalid != TFB_OK) {
        size_t len = tfb_last_error(nullptr, 0);
        plan->why.resize(len + 1);
        tfb_last_error(plan->why.data(), plan->why.size());
        return TFB_OK;
    }
    return lay_out(ctx, dtype, n, problems, balance, &plan->units);
}

tfb_status run(tfb_grouped_plan* plan, tfb::Scalar alpha, tfb::Scalar beta) {
    using namespace tfb;
    if (plan->invalid != TFB_OK) return fail(plan->invalid, "%s", plan->why.c_str());
    DeviceGuard g(plan->ctx->device);
    if (!plan->fast) return run_units(plan->ctx, plan->dtype, plan->units, alpha, beta);
    if (plan->schedule.tcgen05) return grouped_tcgen05_run(plan->ctx, plan->schedule, alpha, beta);
    return grouped_tf32_run(plan->ctx, plan->schedule, alpha, beta);
}

tfb_status check_args(const char* who, tfb_ctx* ctx, int32_t dtype, size_t n, const tfb_gemm_problem* problems) {
    using namespace tfb;
    if (!ctx) return fail(TFB_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", who);
    if (!dtype_valid(dtype)) return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", (int)dtype);
    if (n && !problems) return fail(TFB_ERR_INVALID_ARGUMENT, "%s: problems is NULL", who);
    return TFB_OK;
}

}  // namespace

extern "C" tfb_status tfb_grouped_gemm(tfb_ctx* ctx, int32_t dtype, size_t n_problems, const tfb_gemm_problem* problems,
                                       const void* alpha, const void* beta) {
    using namespace tfb;
    TFB_TRY(check_args("tfb_grouped_gemm", ctx, dtype, n_problems, problems));
    if (!alpha || !beta) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_grouped_gemm: alpha/beta are NULL");
    tfb_grouped_plan plan;
    TFB_TRY(prepare(ctx, dtype, n_problems, problems, false, &plan));
    TFB_TRY(run(&plan, load_scalar(dtype, alpha), load_scalar(dtype, beta)));
    for (PoolBlock* b : {&plan.schedule.mem, &plan.units.mem}) b->keep_for_graph();  // a replay reads the table again
    return TFB_OK;
}

extern "C" tfb_status tfb_grouped_plan_create(tfb_ctx* ctx, int32_t dtype, size_t n_problems,
                                              const tfb_gemm_problem* problems, tfb_grouped_plan** out) {
    using namespace tfb;
    TFB_TRY(check_args("tfb_grouped_plan_create", ctx, dtype, n_problems, problems));
    if (!out) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_grouped_plan_create: out is NULL");
    auto* plan = new (std::nothrow) tfb_grouped_plan;
    if (!plan) return fail(TFB_ERR_DEVICE, "out of host memory");
    const tfb_status st = prepare(ctx, dtype, n_problems, problems, true, plan);
    if (st != TFB_OK) {
        delete plan;
        return st;
    }
    *out = plan;
    return TFB_OK;
}

extern "C" tfb_status tfb_grouped_plan_execute(tfb_grouped_plan* plan, const void* alpha, const void* beta) {
    using namespace tfb;
    if (!plan) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_grouped_plan_execute: plan is NULL");
    if (!alpha || !beta) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_grouped_plan_execute: alpha/beta are NULL");
    return run(plan, load_scalar(plan->dtype, alpha), load_scalar(plan->dtype, beta));
}

extern "C" void tfb_grouped_plan_destroy(tfb_grouped_plan* plan) { delete plan; }
