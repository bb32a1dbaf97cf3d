// Contraction driver: offset tables, kernel selection, and the SIMT kernel that takes
// whatever the tensor-core kernels decline.  Implements the arithmetic of
// `PrimDescriptor::{Contract, BatchedGemm}` (tenferro-prims/src/lib.rs:156-168, 227-239).
#include "contract_common.cuh"
#include "contract_tables.h"
#include "ptx_sm100.cuh"
#include "scalar_ops.cuh"

namespace tfb {

static int64_t prod(const std::vector<Mode>& v) {
    int64_t p = 1;
    for (auto& m : v) p *= m.extent;
    return p;
}
int64_t ContractProblem::M() const { return prod(m); }
int64_t ContractProblem::N() const { return prod(n); }
int64_t ContractProblem::K() const { return prod(k); }
int64_t ContractProblem::B() const { return prod(batch); }

// ------------------------------------------------------------------ offset tables
struct TableJob {
    LoopNest nest;     // the group's modes, strides for tensors 0..2
    int64_t* out[3];   // table per tensor (nullptr: tensor does not carry this group)
};
struct TableJobs {
    TableJob job[4];
};

__global__ void __launch_bounds__(256) build_tables_kernel(TableJobs jobs) {
    const TableJob& j = jobs.job[blockIdx.y];
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < j.nest.total; idx += stride) {
        int64_t rem = idx, off0 = 0, off1 = 0, off2 = 0;
        for (int d = 0; d < j.nest.rank; ++d) {
            int64_t q = rem / j.nest.extent[d];
            int64_t r = rem - q * j.nest.extent[d];
            off0 += r * j.nest.stride[0][d];
            off1 += r * j.nest.stride[1][d];
            off2 += r * j.nest.stride[2][d];
            rem = q;
        }
        if (j.out[0]) j.out[0][idx] = off0;
        if (j.out[1]) j.out[1][idx] = off1;
        if (j.out[2]) j.out[2][idx] = off2;
    }
}

ContractTables::~ContractTables() {
    if (block) cudaFree(block);
    if (built) cudaEventDestroy(built);
}

static std::string signature(const ContractProblem& p) {
    std::string s;
    auto put = [&](const std::vector<Mode>& g) {
        int64_t n = (int64_t)g.size();
        s.append((const char*)&n, sizeof n);
        for (auto& m : g) s.append((const char*)&m, sizeof m);
    };
    put(p.batch);
    put(p.m);
    put(p.n);
    put(p.k);
    s.push_back(p.mul ? 'd' : '-');
    return s;
}

struct TableCache {
    std::mutex mu;
    std::map<std::pair<int, std::string>, std::shared_ptr<ContractTables>> map;
    std::vector<std::pair<int, std::string>> order;
};
static TableCache& cache() {
    static TableCache c;
    return c;
}

tfb_status get_tables(tfb_ctx* ctx, const ContractProblem& p, std::shared_ptr<ContractTables>* out) {
    auto key = std::make_pair(ctx->device, signature(p));
    TableCache& tc = cache();
    std::lock_guard<std::mutex> lock(tc.mu);
    auto it = tc.map.find(key);
    if (it != tc.map.end()) {
        ContractTables& hit = *it->second;
        // Same stream as the build: stream order is enough.  Any other stream (another context
        // of this device, or this context after tfb_ctx_set_stream) must not read the tables
        // before the kernels that fill them have run.
        if (!hit.ready && hit.built) {
            if (cudaEventQuery(hit.built) == cudaSuccess) {
                hit.ready = true;
            } else {
                cudaGetLastError();
                if (ctx->stream != hit.build_stream) TFB_CUDA(cudaStreamWaitEvent(ctx->stream, hit.built, 0));
            }
        }
        *out = it->second;
        return TFB_OK;
    }
    auto t = std::make_shared<ContractTables>();
    t->M = p.M();
    t->N = p.N();
    t->K = p.K();
    t->B = p.B();
    // One allocation: a_b b_b c_b | a_m c_m | b_n c_n | a_k b_k | d_b d_m d_n
    size_t n_entries = (size_t)(3 * t->B + 2 * t->M + 2 * t->N + 2 * t->K);
    if (p.mul) n_entries += (size_t)(t->B + t->M + t->N);
    TFB_CUDA(cudaMalloc(&t->block, n_entries * sizeof(int64_t) + 64));
    int64_t* q = (int64_t*)t->block;
    t->a_b = q; q += t->B;
    t->b_b = q; q += t->B;
    t->c_b = q; q += t->B;
    t->a_m = q; q += t->M;
    t->c_m = q; q += t->M;
    t->b_n = q; q += t->N;
    t->c_n = q; q += t->N;
    t->a_k = q; q += t->K;
    t->b_k = q; q += t->K;
    if (p.mul) {
        t->d_b = q; q += t->B;
        t->d_m = q; q += t->M;
        t->d_n = q; q += t->N;
    }
    TableJobs jobs;
    TFB_TRY(make_nest(p.batch, &jobs.job[0].nest));
    jobs.job[0].out[0] = t->a_b; jobs.job[0].out[1] = t->b_b; jobs.job[0].out[2] = t->c_b;
    TFB_TRY(make_nest(p.m, &jobs.job[1].nest));
    jobs.job[1].out[0] = t->a_m; jobs.job[1].out[1] = nullptr; jobs.job[1].out[2] = t->c_m;
    TFB_TRY(make_nest(p.n, &jobs.job[2].nest));
    jobs.job[2].out[0] = nullptr; jobs.job[2].out[1] = t->b_n; jobs.job[2].out[2] = t->c_n;
    TFB_TRY(make_nest(p.k, &jobs.job[3].nest));
    jobs.job[3].out[0] = t->a_k; jobs.job[3].out[1] = t->b_k; jobs.job[3].out[2] = nullptr;
    int64_t biggest = std::max(std::max(t->B, t->M), std::max(t->N, t->K));
    int gx = (int)std::min<int64_t>((biggest + 255) / 256, 1024);
    if (gx < 1) gx = 1;
    LaunchScope ls(ctx, "build_tables");
    build_tables_kernel<<<dim3(gx, 4), 256, 0, ctx->stream>>>(jobs);
    TFB_CUDA(cudaGetLastError());
    if (p.mul) {
        // The multiplier's offsets over the same three output groups (its strides are slot 3).
        auto slot3 = [](const std::vector<Mode>& g) {
            std::vector<Mode> r;
            for (auto& m : g) r.push_back(Mode{m.extent, {m.s[3], 0, 0}});
            return r;
        };
        TableJobs dj;
        TFB_TRY(make_nest(slot3(p.batch), &dj.job[0].nest));
        TFB_TRY(make_nest(slot3(p.m), &dj.job[1].nest));
        TFB_TRY(make_nest(slot3(p.n), &dj.job[2].nest));
        TFB_TRY(make_nest(std::vector<Mode>{}, &dj.job[3].nest));
        dj.job[3].nest.total = 0;
        for (int j = 0; j < 4; ++j) dj.job[j].out[0] = dj.job[j].out[1] = dj.job[j].out[2] = nullptr;
        dj.job[0].out[0] = t->d_b;
        dj.job[1].out[0] = t->d_m;
        dj.job[2].out[0] = t->d_n;
        build_tables_kernel<<<dim3(gx, 4), 256, 0, ctx->stream>>>(dj);
        count_launch();
        TFB_CUDA(cudaGetLastError());
    }
    TFB_CUDA(cudaEventCreateWithFlags(&t->built, cudaEventDisableTiming));
    TFB_CUDA(cudaEventRecord(t->built, ctx->stream));
    t->build_stream = ctx->stream;
    // Bounded cache: drop the oldest entry once 256 layouts are held.  Tables in use by
    // enqueued kernels stay alive through cudaFree's implicit synchronisation.
    if (tc.order.size() >= 256) {
        tc.map.erase(tc.order.front());
        tc.order.erase(tc.order.begin());
    }
    tc.map[key] = t;
    tc.order.push_back(key);
    *out = t;
    return TFB_OK;
}

// Unit-stride analysis of one operand tile: is the group's first (fastest) mode stride 1 in
// tensor `t`, and can two f64 travel as one 16-byte chunk?
static bool group_unit_stride(const std::vector<Mode>& g, int t) { return !g.empty() && g[0].s[t] == 1; }
static bool all_even(const std::vector<Mode>& g, int t, size_t from) {
    for (size_t i = from; i < g.size(); ++i)
        if (g[i].s[t] % 2 != 0) return false;
    return true;
}

void fill_args(const ContractProblem& p, const ContractTables* tables, ContractArgs* a) {
    memset(a, 0, sizeof *a);
    a->a = (const char*)p.a;
    a->b = (const char*)p.b;
    a->c = (char*)p.c;
    if (tables) {
        const ContractTables& t = *tables;
        a->a_b = t.a_b; a->b_b = t.b_b; a->c_b = t.c_b;
        a->a_m = t.a_m; a->c_m = t.c_m;
        a->b_n = t.b_n; a->c_n = t.c_n;
        a->a_k = t.a_k; a->b_k = t.b_k;
        a->d_b = t.d_b; a->d_m = t.d_m; a->d_n = t.d_n;
    }
    a->M = p.M(); a->N = p.N(); a->K = p.K(); a->B = p.B();
    auto step = [](const std::vector<Mode>& g, int slot) { return g.empty() ? (int64_t)0 : g[0].s[slot]; };
    a->c_bs = step(p.batch, 2); a->c_ms = step(p.m, 2); a->c_ns = step(p.n, 2);
    a->d_bs = step(p.batch, 3); a->d_ms = step(p.m, 3); a->d_ns = step(p.n, 3);
    a->alpha_re = p.alpha.re; a->alpha_im = p.alpha.im;
    a->beta_re = p.beta.re; a->beta_im = p.beta.im;
    a->conj_a = p.conj_a && dtype_is_complex(p.dtype);
    a->conj_b = p.conj_b && dtype_is_complex(p.dtype);
    a->mul = (const char*)p.mul;
    a->conj_mul = p.conj_mul && dtype_is_complex(p.dtype);
    // Direction of the unit stride in each operand tile.  If neither group is unit-stride
    // the choice only affects which threads sit next to each other.
    bool a_k1 = group_unit_stride(p.k, 0), a_m1 = group_unit_stride(p.m, 0);
    bool b_k1 = group_unit_stride(p.k, 1), b_n1 = group_unit_stride(p.n, 1);
    a->a_kfast = a_k1 || !a_m1;
    a->b_kfast = b_k1 || !b_n1;
    a->a_vec = a->b_vec = 1;
    if (p.dtype == TFB_F64) {
        // 16-byte chunks of two doubles along the unit-stride group: its first extent must be
        // even, every other stride of that operand even, and the element pointer 16-byte aligned.
        auto pair_ok = [&](const std::vector<Mode>& fast, const std::vector<Mode>& other, int tns, const void* base) {
            if (fast.empty() || fast[0].s[tns] != 1 || fast[0].extent % 2 != 0) return false;
            if (!all_even(fast, tns, 1) || !all_even(other, tns, 0) || !all_even(p.batch, tns, 0)) return false;
            return (uintptr_t)base % 16 == 0;
        };
        if (a->a_kfast ? pair_ok(p.k, p.m, 0, p.a) : pair_ok(p.m, p.k, 0, p.a)) a->a_vec = 2;
        if (a->b_kfast ? pair_ok(p.k, p.n, 1, p.b) : pair_ok(p.n, p.k, 1, p.b)) a->b_vec = 2;
    }
}

// ------------------------------------------------------------------ SIMT kernel
// Exact in the element type (FMA), any strides, any dtype: the path of what the tensor-core kernels
// decline or would mostly pad - f32 and complex32 outputs with a short side, f32 layouts TMA cannot describe
// below the size that repays a copy - and of the tropical semirings (ALG, scalar_ops.cuh: the same
// loop nest computes C = alpha (x) (+)_k A (x) B  (+)  beta (x) C).
//
// 64 x 64 block tile, 16-deep k slices (8 for 16-byte elements), 256 threads, 4 x 4 outputs each.  The next
// slice is in flight from global memory to registers while one is computed from shared memory, and a
// f32 fragment is four neighbours, one 16-byte access.  Few tiles with a long K are cut into
// gridDim.y ranges whose sums simt_finish_kernel adds in range order (no result depends on timing).
// Small shapes are bound by latency, the rest by issue and shared memory (kernel and finish): 679 x 636 x 431 f32
// 90 -> 33 us, 510 x 690 x 945 105 -> 48, 38 x 1209 x 31 complex32 240 -> 33 (one tile, so one CTA before),
// 202 x 150 x 70 f32 27 -> 22.
template <typename T>
constexpr int kSimtK = sizeof(T) == 16 ? 8 : 16;
template <typename T>
constexpr int kSimtCtas = sizeof(T) == 4 ? 3 : sizeof(T) == 16 ? 1 : 2;  // CTAs per SM (f32 spills 84 bytes at three)

// beta equal to the semiring's zero means "overwrite": the output is never read.
template <int ALG>
__device__ __forceinline__ bool simt_reads_c(const ContractArgs& g) {
    return ALG == 0 ? (g.beta_re != 0 || g.beta_im != 0) : !(g.beta_re == (ALG == 1 ? -INFINITY : INFINITY));
}
// `old`: what the output holds, where it is read.
template <typename T, int ALG>
__device__ __forceinline__ T simt_result(const ContractArgs& g, const T* D, int64_t m, int64_t n, T old, T sum) {
    using S = Semi<T, ALG>;
    if (D) {
        const T d = D[g.d_m[m] + g.d_n[n]];
        sum = Ops<T>::mul(sum, g.conj_mul ? Ops<T>::conj(d) : d);
    }
    const T v = S::mul(Ops<T>::from(Scalar{g.alpha_re, g.alpha_im}), sum);
    return simt_reads_c<ALG>(g) ? S::add(v, S::mul(Ops<T>::from(Scalar{g.beta_re, g.beta_im}), old)) : v;
}

template <typename T, int ALG = 0>
__global__ void __launch_bounds__(256, kSimtCtas<T>) contract_simt_kernel(ContractArgs g) {
    launch_begin();
    using S = Semi<T, ALG>;
    constexpr int BM = 64, BN = 64, BK = kSimtK<T>, P = 68, L = BM * BK / 256;
    // A thread's fragment: four neighbours for 4-byte elements, else four 16 apart, which meet no bank twice (988 x
    // 1383 x 127 complex double 165 us with neighbours, 111 without) and leave a small output to more threads.
    constexpr int E = sizeof(T) > 4 ? 1 : 4, J = sizeof(T) > 4 ? 16 : 1;
    __shared__ __align__(16) T As[2][BK][P];
    __shared__ __align__(16) T Bs[2][BK][P];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, each 4 x 4
    // A thread's L elements of each operand slice: neighbouring threads follow the unit stride.
    int am[L], ak[L], bn[L], bk[L];
#pragma unroll
    for (int r = 0; r < L; ++r) {
        const int c = tid + r * 256;
        if (g.a_kfast) { ak[r] = c % BK; am[r] = c / BK; } else { am[r] = c % BM; ak[r] = c / BM; }
        if (g.b_kfast) { bk[r] = c % BK; bn[r] = c / BK; } else { bn[r] = c % BN; bk[r] = c / BN; }
    }
    const int64_t s0 = (int64_t)blockIdx.y * g.iters_per_cta, s1 = min(g.k_iters, s0 + g.iters_per_cta);
    for (int64_t tile = blockIdx.x; tile < g.n_tiles; tile += gridDim.x) {
        const int64_t tm = tile % g.tiles_m, rest = tile / g.tiles_m, tn = rest % g.tiles_n, bb = rest / g.tiles_n;
        const int64_t m0 = tm * BM, n0 = tn * BN;
        const T* Ab = (const T*)g.a + g.a_b[bb];
        const T* Bb = (const T*)g.b + g.b_b[bb];
        int64_t arow[L], brow[L];
#pragma unroll
        for (int r = 0; r < L; ++r) {
            arow[r] = m0 + am[r] < g.M ? g.a_m[m0 + am[r]] : 0;
            brow[r] = n0 + bn[r] < g.N ? g.b_n[n0 + bn[r]] : 0;
        }
        T va[L], vb[L];
        auto fetch = [&](int64_t slice) {
            const int64_t k0 = slice * BK;
#pragma unroll
            for (int r = 0; r < L; ++r) {
                va[r] = vb[r] = S::zero();
                if (m0 + am[r] < g.M && k0 + ak[r] < g.K) va[r] = Ab[arow[r] + g.a_k[k0 + ak[r]]];
                if (n0 + bn[r] < g.N && k0 + bk[r] < g.K) vb[r] = Bb[brow[r] + g.b_k[k0 + bk[r]]];
            }
        };
        auto put = [&](int buf) {
#pragma unroll
            for (int r = 0; r < L; ++r) {
                As[buf][ak[r]][am[r]] = g.conj_a ? Ops<T>::conj(va[r]) : va[r];
                Bs[buf][bk[r]][bn[r]] = g.conj_b ? Ops<T>::conj(vb[r]) : vb[r];
            }
        };
        T acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = S::zero();
        if (s0 < s1) {
            fetch(s0);
            put(0);
        }
        __syncthreads();
        int buf = 0;
        for (int64_t s = s0; s < s1; ++s, buf ^= 1) {
            if (s + 1 < s1) fetch(s + 1);
#pragma unroll 4
            for (int kk = 0; kk < BK; ++kk) {
                T av[4], bv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) av[i] = As[buf][kk][E * tx + J * i];
#pragma unroll
                for (int j = 0; j < 4; ++j) bv[j] = Bs[buf][kk][E * ty + J * j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = S::fma_(av[i], bv[j], acc[i][j]);
            }
            if (s + 1 < s1) put(buf ^ 1);
            __syncthreads();
        }
        if (g.partial) {
            T* P0 = (T*)g.partial + ((int64_t)blockIdx.y * g.n_tiles + tile) * (BM * BN);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) P0[(E * ty + J * j) * BM + E * tx + J * i] = acc[i][j];
            continue;
        }
        T* Cb = (T*)g.c + g.c_b[bb];
        const T* D = g.mul ? reinterpret_cast<const T*>(g.mul) + g.d_b[bb] : nullptr;
        // A thread's outputs are read together, not one after the other's store.
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t n = n0 + E * ty + J * j;
            if (n >= g.N) continue;
            T* col = Cb + g.c_n[n];
            T old[4];
            if (simt_reads_c<ALG>(g)) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int64_t m = m0 + E * tx + J * i;
                    if (m < g.M) old[i] = col[g.c_m[m]];
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t m = m0 + E * tx + J * i;
                if (m < g.M) col[g.c_m[m]] = simt_result<T, ALG>(g, D, m, n, old[i], acc[i][j]);
            }
        }
    }
}

// Adds the ranges of each output element in range order; one thread per element of a tile.
template <typename T, int ALG = 0>
__global__ void __launch_bounds__(256) simt_finish_kernel(ContractArgs g, int splits) {
    launch_begin();
    constexpr int BM = 64, BN = 64;
    const int64_t tile = blockIdx.x, tm = tile % g.tiles_m, rest = tile / g.tiles_m, tn = rest % g.tiles_n, bb = rest / g.tiles_n;
    const int e = blockIdx.y * 256 + threadIdx.x;
    const int64_t m = tm * BM + e % BM, n = tn * BN + e / BM;
    if (m >= g.M || n >= g.N) return;
    const T* P0 = (const T*)g.partial + tile * (BM * BN) + e;
    T sum = P0[0];
#pragma unroll 8
    for (int s = 1; s < splits; ++s) sum = Semi<T, ALG>::add(sum, P0[(int64_t)s * g.n_tiles * (BM * BN)]);
    T* at = (T*)g.c + g.c_b[bb] + g.c_m[m] + g.c_n[n];
    const T old = simt_reads_c<ALG>(g) ? *at : sum;
    *at = simt_result<T, ALG>(g, g.mul ? reinterpret_cast<const T*>(g.mul) + g.d_b[bb] : nullptr, m, n, old, sum);
}

template <typename T, int ALG>
static tfb_status simt_launch(tfb_ctx* ctx, ContractArgs a, const char* name) {
    constexpr int BK = kSimtK<T>;
    a.tiles_m = (a.M + 63) / 64;
    a.tiles_n = (a.N + 63) / 64;
    a.n_tiles = a.tiles_m * a.tiles_n * a.B;
    if (a.n_tiles == 0) return TFB_OK;
    a.k_iters = (a.K + BK - 1) / BK;
    // As many ranges as run at once; a range keeps at least eight slices, below which the finishing launch
    // costs more than it saves.
    int64_t splits = std::min<int64_t>((int64_t)ctx->sm_count * kSimtCtas<T> / a.n_tiles, a.k_iters / 8);
    splits = std::max<int64_t>(1, std::min<int64_t>(splits, 64));
    PoolBlock ws;
    // Without room for the sums the ranges stay whole, as the call must not need memory to succeed.
    if (splits > 1 && ws.alloc(ctx, (size_t)(splits * a.n_tiles) * 64 * 64 * sizeof(T)) != TFB_OK) splits = 1;
    a.iters_per_cta = (a.k_iters + splits - 1) / splits;
    if (splits > 1) splits = (a.k_iters + a.iters_per_cta - 1) / a.iters_per_cta;
    a.partial = splits > 1 ? (char*)ws.ptr : nullptr;
    const unsigned grid = (unsigned)std::min<int64_t>(a.n_tiles, (int64_t)ctx->sm_count * 8);
    {
        LaunchScope ls(ctx, name);
        TFB_CUDA(launch_overlapped(ctx, contract_simt_kernel<T, ALG>, dim3(grid, (unsigned)splits), dim3(256), 0, 0u, a));
    }
    if (splits > 1) {
        LaunchScope ls(ctx, "contract_simt_finish");
        TFB_CUDA(launch_overlapped(ctx, simt_finish_kernel<T, ALG>, dim3((unsigned)a.n_tiles, 16), dim3(256), 0, 0u, a, (int)splits));
    }
    return TFB_OK;
}

tfb_status contract_simt(tfb_ctx* ctx, const ContractProblem& p) {
    std::shared_ptr<ContractTables> t;
    TFB_TRY(get_tables(ctx, p, &t));
    ContractArgs a;
    fill_args(p, t.get(), &a);
    switch (p.dtype) {
        case TFB_F32: return simt_launch<float, 0>(ctx, a, "contract_simt");
        case TFB_F64: return simt_launch<double, 0>(ctx, a, "contract_simt");
        case TFB_C32: return simt_launch<float2, 0>(ctx, a, "contract_simt");
        case TFB_C64: return simt_launch<double2, 0>(ctx, a, "contract_simt");
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", p.dtype);
}

// The same kernel over a non-Standard semiring (real types only): 1 MaxPlus, 2 MinPlus.
tfb_status contract_simt_semiring(tfb_ctx* ctx, const ContractProblem& p, int algebra) {
    if (p.dtype != TFB_F32 && p.dtype != TFB_F64)
        return fail(TFB_ERR_INVALID_ARGUMENT, "MaxPlus and MinPlus are defined for f32 and f64");
    if (p.mul) return fail(TFB_ERR_INVALID_ARGUMENT, "a fused multiplier is a Standard-algebra feature");
    DeviceGuard guard(ctx->device);
    std::shared_ptr<ContractTables> t;
    TFB_TRY(get_tables(ctx, p, &t));
    ContractArgs a;
    fill_args(p, t.get(), &a);
    const char* name = "contract_simt_semiring";
    if (p.dtype == TFB_F32 && algebra == 1) return simt_launch<float, 1>(ctx, a, name);
    if (p.dtype == TFB_F32 && algebra == 2) return simt_launch<float, 2>(ctx, a, name);
    if (p.dtype == TFB_F64 && algebra == 1) return simt_launch<double, 1>(ctx, a, name);
    if (p.dtype == TFB_F64 && algebra == 2) return simt_launch<double, 2>(ctx, a, name);
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown algebra %d", algebra);
}

// ------------------------------------------------------------------ batch index innermost
// "bij,bjk->bik" in column-major order: neighbouring elements of the output belong to different products, so a kernel that
// writes a tile of one of them touches a 32-byte sector per element, and reads its operands the same way.  From
// the size on that repays copies at all, the operands that lie so are copied with the batch outermost, the
// products go to a block of their own, and one pass over that applies alpha and beta and puts the batch back innermost: all
// of it tiled permutations at the memory's rate.
// (us as they lie and on copies: f32, 100 of 900^3 4560, 1140, the exact kernel 1000 of 100^3 380, 233, 8 of 600^3 255, 227, 477 of 100
// x 800 x 17 576, 386; double, 220 of 580 x 308 x 408 2340, 1540, 100 of 500 x 500 x 16 838, 167, 16 of 600^3 357, 334; complex
// single, 1000 of 100^3 332, 260, 100 of 500 x 500 x 16 456, 186.  Complex double elements are half a sector, and nothing is gained:
// 64 of 300^3 619, 628.)
static tfb_status contract_batch_innermost(tfb_ctx* ctx, const ContractProblem& p, const char** used, bool* done) {
    *done = false;
    if (p.batch.size() != 1 || p.batch[0].s[2] != 1 || p.mul || p.dtype == TFB_C64) return TFB_OK;
    if (p.batch[0].extent < (p.dtype == TFB_F32 ? 8 : p.dtype == TFB_F64 ? 16 : 32)) return TFB_OK;
    if (p.dtype == TFB_F32 && p.k.size() > 2) return TFB_OK;  // the exact kernel's, as are those below
    const int64_t M = p.M(), N = p.N(), K = p.K(), B = p.B(), es = (int64_t)dtype_size(p.dtype);
    const bool wide = p.dtype == TFB_F64;
    const double flops = (dtype_is_complex(p.dtype) ? 8.0 : 2.0) * (double)M * (double)N * (double)K * (double)B;
    if (M < 64 || N < 64 || K < 16 || flops < (wide ? 2e8 : 1e9)) return TFB_OK;
    // Long and thin outputs of a short K are bound by their own passes (436 of 105 x 817 x 17 complex single: 874 us as they lie, 1069
    // on copies; 100 of 500 x 500 x 16 444, 186).
    if (p.dtype == TFB_C32 && K < 32 && std::max(M, N) > 5 * std::min(M, N)) return TFB_OK;
    auto up = [](int64_t x, int64_t to) { return (x + to - 1) / to * to; };
    // Copies as the kernels like them best: [batch][k][rows] for the FP64 pipe, [batch][rows][k] for tcgen05.  The first operand of
    // a complex single product is embedded from either, and by rows it does not offer itself to be read in place with the
    // roles exchanged, which would take rows across the block (488 of 260 x 80 x 16: 286 us exchanged, 133 so,
    // 148 as they lie).
    const bool copy[2] = {p.batch[0].s[0] == 1, p.batch[0].s[1] == 1};
    // A batch index innermost leaves an operand without a tensor map, and contract_tcgen05 copies those of large products only:
    // smaller ones run on the exact kernel, and do so on the copies (relative error of 1000 of 100^3 1.8e-7, as 3xTF32 8.7e-7).
    const bool exact = p.dtype == TFB_F32 && (copy[0] || copy[1]) && 2.0 * (double)M * (double)N * (double)K < kTcCopyFlops;
    // Double precision products whose output stays in L2 find the sectors of their stores there: nothing to gain where an operand is
    // read in place besides (115 of 784 x 64 x 112, 46 MB: 85 us as they lie, 97 on copies; 533 of them 1105, 376).
    if (wide && !(copy[0] && copy[1]) && (double)M * (double)N * (double)B * (double)es < 80e6) return TFB_OK;
    const bool by_rows[2] = {p.dtype != TFB_F32, wide};
    const int64_t rows[2] = {M, N};
    int64_t ld[3], per[3], bytes = 0;
    for (int t = 0; t < 2; ++t) {
        ld[t] = by_rows[t] ? up(rows[t], 8) : up(K, 4);
        per[t] = ld[t] * (by_rows[t] ? K : rows[t]);
        if (copy[t]) bytes += per[t] * es;
    }
    ld[2] = up(M, 8);
    per[2] = ld[2] * up(N, 8);
    bytes += per[2] * es;
    // Copies of as many products as a gigabyte holds, whole sectors of the batch (eight) at least: the pool keeps the memory, and more
    // than a thirty-second of the device's (5.7 GB), as for the copies of a double precision product, is not asked for.
    const int64_t most = env_int("TFB_BATCH_CHUNK", 0) > 0 ? env_int("TFB_BATCH_CHUNK", 0) : ((int64_t)1 << 30) / bytes;
    const int64_t chunk = std::min(B, std::max<int64_t>(8, most >= 32 ? most / 32 * 32 : most / 8 * 8));
    if ((double)bytes * (double)chunk > (double)ctx->total_mem / 32) return TFB_OK;
    auto dense = [](std::vector<Mode>& g, int t, int64_t step) {
        for (Mode& m : g) {
            m.s[t] = step;
            step *= m.extent;
        }
    };
    // The product of n of the batch on the copies, and the nests of the passes that make them and put its output back;
    // false where a pass has more modes than a nest takes, though each group of the product alone has not.
    auto lay_out = [&](int64_t n, ContractProblem* q, LoopNest* nest) -> bool {
        *q = p;
        q->batch[0].extent = n;
        for (int t = 0; t < 3; ++t) {
            if (t < 2 && !copy[t]) continue;
            std::vector<Mode> modes;
            // from where the operand lies to its copy, from the block to where the output lies
            auto put = [&](const std::vector<Mode>& outer, const std::vector<Mode>& block) {
                for (size_t i = 0; i < block.size(); ++i)
                    modes.push_back(t < 2 ? Mode{block[i].extent, {outer[i].s[t], block[i].s[t], 0, 0}}
                                          : Mode{block[i].extent, {block[i].s[t], outer[i].s[t], 0, 0}});
            };
            if (t < 2) {
                std::vector<Mode>& free_q = t == 0 ? q->m : q->n;
                dense(free_q, t, by_rows[t] ? 1 : ld[t]);
                dense(q->k, t, by_rows[t] ? ld[t] : 1);
                put(t == 0 ? p.m : p.n, free_q);
                put(p.k, q->k);
            } else {
                dense(q->m, 2, 1);
                dense(q->n, 2, ld[2]);
                put(p.m, q->m);
                put(p.n, q->n);
            }
            q->batch[0].s[t] = per[t];
            put(p.batch, q->batch);
            sort_and_fuse(modes, 1, 2);
            if ((int)modes.size() > kMaxRank || make_nest(modes, &nest[t]) != TFB_OK) return false;
        }
        for (auto* g : {&q->m, &q->n, &q->k}) fuse_in_order(*g, 4);
        // rows of a copy are a multiple of eight, which its tensor map asks for: those past the last are products of
        // whatever lies there, and land between the block's columns
        if (wide && copy[0]) q->m.assign(1, Mode{ld[0], {1, 0, 1, 0}});
        if (wide && copy[1]) q->n.assign(1, Mode{ld[1], {0, 1, ld[2], 0}});
        return true;
    };
    ContractProblem q;
    LoopNest nest[3];
    for (int64_t n : {B % chunk, chunk})
        if (n > 0 && !lay_out(n, &q, nest)) return TFB_OK;
    PoolBlock blk[3];
    for (int t = 0; t < 3; ++t)
        if ((t == 2 || copy[t]) && blk[t].alloc(ctx, (size_t)(per[t] * chunk * es)) != TFB_OK) return TFB_OK;
    for (int64_t b0 = 0; b0 < B; b0 += chunk) {
        lay_out(std::min(chunk, B - b0), &q, nest);
        q.a = (const char*)p.a + b0 * p.batch[0].s[0] * es;
        q.b = (const char*)p.b + b0 * p.batch[0].s[1] * es;
        q.c = blk[2].ptr;
        q.alpha = Scalar{1.0, 0.0};
        q.beta = Scalar{0.0, 0.0};
        for (int t = 0; t < 2; ++t) {
            if (!copy[t]) continue;
            const void*& x = t == 0 ? q.a : q.b;
            TFB_TRY(launch_permute(ctx, p.dtype, nest[t], x, blk[t].ptr, Scalar{1.0, 0.0}, Scalar{0.0, 0.0}, false));
            x = blk[t].ptr;
        }
        const tfb_status st = launch_contract(ctx, q, exact ? CK_SIMT : CK_AUTO, used);
        if (st != TFB_OK) return b0 == 0 ? TFB_OK : st;  // no room for its scratch beside the copies: as the operands lie
        TFB_TRY(launch_permute(ctx, p.dtype, nest[2], blk[2].ptr, (char*)p.c + b0 * es, p.alpha, p.beta, false));
    }
    *done = true;
    return TFB_OK;
}

// ------------------------------------------------------------------ selection
tfb_status launch_contract(tfb_ctx* ctx, const ContractProblem& p, int force_kernel, const char** used) {
    DeviceGuard g(ctx->device);
    if (used) *used = "none";
    const int64_t M = p.M(), N = p.N(), K = p.K(), B = p.B();
    if (M == 0 || N == 0 || B == 0) return TFB_OK;  // empty output
    if (K == 0) {
        // Empty sum: C = beta * C.
        std::vector<Mode> modes;
        for (auto* grp : {&p.batch, &p.m, &p.n})
            for (auto& m : *grp) modes.push_back(Mode{m.extent, {m.s[2], 0, 0}});
        LoopNest nest;
        TFB_TRY(make_nest(modes, &nest));
        if (used) *used = "scale";
        return launch_scale(ctx, p.dtype, nest, p.c, p.beta);
    }
    int want = force_kernel != CK_AUTO ? force_kernel : env_int("TFB_FORCE_KERNEL", CK_AUTO);
    bool declined = false;
    if (want == CK_AUTO && env_int("TFB_BATCH_OUTERMOST", 1)) {
        bool done = false;
        TFB_TRY(contract_batch_innermost(ctx, p, used, &done));
        if (done) return TFB_OK;
    }
    if (want == CK_AUTO || want == CK_TCGEN05) {
        if (p.dtype == TFB_F32 || p.dtype == TFB_C32) {
            if (p.dtype == TFB_C32)
                TFB_TRY(contract_c32_embedded(ctx, p, &declined));
            else
                TFB_TRY(contract_tcgen05(ctx, p, &declined));
            if (!declined) {
                if (used) *used = "tcgen05_tf32x3";
                return TFB_OK;
            }
            if (want == CK_TCGEN05)
                return fail(TFB_ERR_INVALID_ARGUMENT, "tcgen05 kernel forced but it cannot stage this layout");
        } else if (want == CK_TCGEN05) {
            return fail(TFB_ERR_INVALID_ARGUMENT, "tcgen05 kernel forced but the dtype is not f32/c32");
        }
    }
    if (want == CK_AUTO || want == CK_DMMA || want == CK_DMMA4) {
        if (p.dtype == TFB_F64 || p.dtype == TFB_C64) {
            const bool four = want == CK_DMMA4 || env_int("TFB_C64_FOUR_PRODUCTS", 0) != 0;
            TFB_TRY(contract_dmma(ctx, p, &declined, four));
            if (!declined) {
                if (used) *used = "dmma_f64";
                return TFB_OK;
            }
        } else if (want == CK_DMMA || want == CK_DMMA4) {
            return fail(TFB_ERR_INVALID_ARGUMENT, "DMMA kernel forced but the dtype is not f64/c64");
        }
    }
    if (used) *used = "simt";
    return contract_simt(ctx, p);
}

}  // namespace tfb
