// Complex32 contraction on the tensor cores as ONE real 3xTF32 product.
//
// A complex product is a real product of doubled extents:
//
//   [ Re C ]   [ Re A  -Im A ] [ Re B ]
//   [ Im C ] = [ Im A   Re A ] [ Im B ]
//
// With the real and imaginary parts interleaved along the rows of C' (row 2m + c), along K of
// both operands (column 2k + c) this reads  C' (2M x N) = A' (2M x 2K) B' (2K x N),  where
//   * C' is the complex output itself, seen as f32: element (m, n) part c lives at float offset
//     2 * offset(m, n) + c, which the kernel's per-row / per-column offset tables express for
//     ANY output strides - so the product is written straight into C, with no planes to recombine;
//   * B' (stored K-major, [n][2k + c]) is the complex operand copied with K fastest - or, when
//     B already has unit stride along a single contracted mode and no conjugation, B itself;
//   * A' is built once by a gather kernel ([2m + c'][2k + c], K-major) with conjugation and the
//     complex alpha folded in.
// Four real products' worth of MMAs instead of the three of the 3M scheme, but no product
// planes (3 x M x N floats written and read again), no cancellation in the imaginary part, and
// one launch of the f32 kernel whatever the output layout.  A complex beta that is not real is
// applied by scaling C first.  A fused multiplier (ContractProblem::mul) is applied to C in
// place after the product.
//
// Semantics: PrimDescriptor::{Contract, BatchedGemm} for Complex32,
// tenferro-prims/src/lib.rs:156-168, 227-239.
#include <algorithm>

#include "contract_pair.cuh"
#include "contract_tables.h"

namespace tfb {

namespace {

struct EmbedArgs {
    const float2* src;
    const int64_t* row_tab;  // a_m or b_n
    const int64_t* k_tab;
    const int64_t* b_tab;
    int64_t rows, K, B;
    int64_t ld;              // floats per output row (>= 2K, multiple of 4)
    int src_kfast, conj, embed;
    float2 alpha;
    float* dst;              // embed: [B][2 rows][ld], else [B][rows][ld]
};

// The output's offset tables: C seen as f32, row 2m + c -> 2 c_m[m] + c, column n -> 2 c_n[n], batch b -> 2 c_b[b].
struct RealTables {
    const int64_t *c_m, *c_n, *c_b;
    int64_t M, N, B;
    int64_t *out_m, *out_n, *out_b;
};

// 32 x 32 (rows x k) patches through shared memory: reads follow the source's unit stride,
// writes follow k.  embed = 1 writes the 2 x 2 real block of alpha * op(a) per element (two
// output rows), embed = 0 the element itself.  blockIdx.y: the tables, the first operand, the second where it is copied.
// A few MB each, bound by latency: one launch, and a thread's four loads in flight together.  Scattered sources of more than half of
// L2 are bound by sectors that the next product of the batch, or the next patch, finds in L2 again if not too many are on their
// way: one load at a time, and a launch for each operand (400 of 52 x 320 x 880, batch innermost: 2510 us as one launch with
// four loads in flight, 1255 so; 30 of 60^3, which L2 holds, 21 us a call, 26 so).  (Two parameters and a choice rather than an indexed array of them, which is
// read from memory at each use.)
template <bool SCATTERED>
__global__ void __launch_bounds__(256) embed_setup_kernel(EmbedArgs first, EmbedArgs second, RealTables args, int job0, Gate gate) {
    __shared__ float2 tile[32][33];
    launch_begin();
    if (gate.closed()) return;
    const int job = job0 + (int)blockIdx.y;
    if (job == 0) {
        const int64_t n = max(2 * args.M, max(args.N, args.B));
        for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
            if (i < 2 * args.M) args.out_m[i] = 2 * args.c_m[i >> 1] + (i & 1);
            if (i < args.N) args.out_n[i] = 2 * args.c_n[i];
            if (i < args.B) args.out_b[i] = 2 * args.c_b[i];
        }
        return;
    }
    const EmbedArgs g = job == 1 ? first : second;
    const int64_t tiles_r = (g.rows + 31) / 32, tiles_k = (g.K + 31) / 32;
    const int64_t n_tiles = tiles_r * tiles_k * g.B;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int64_t kpad = g.ld / 2;  // complex columns per output row, zero-filled past K
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int64_t tr = t % tiles_r, rest = t / tiles_r, tk = rest % tiles_k, b = rest / tiles_k;
        const int64_t r0 = tr * 32, k0 = tk * 32;
        const float2* src = g.src + g.b_tab[b];
        auto load = [&](int j) {
            // (r, k) of this thread's element: tx runs along the source's fast direction
            const int64_t r = r0 + (g.src_kfast ? j : tx), k = k0 + (g.src_kfast ? tx : j);
            return r < g.rows && k < g.K ? src[g.row_tab[r] + g.k_tab[k]] : make_float2(0.f, 0.f);
        };
        auto put = [&](int j, float2 v) {
            if (g.src_kfast) tile[j][tx] = v; else tile[tx][j] = v;  // tile[r][k]
        };
        if constexpr (SCATTERED) {
#pragma unroll 1
            for (int j = ty; j < 32; j += 8) put(j, load(j));
        } else {
            float2 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = load(ty + 8 * i);
#pragma unroll
            for (int i = 0; i < 4; ++i) put(ty + 8 * i, v[i]);
        }
        __syncthreads();
        for (int j = ty; j < 32; j += 8) {
            const int64_t r = r0 + j, k = k0 + tx;
            if (r < g.rows && k < kpad) {
                float2 v = (k < g.K) ? tile[j][tx] : make_float2(0.f, 0.f);
                if (g.conj) v.y = -v.y;
                if (g.embed) {
                    const float2 w = make_float2(g.alpha.x * v.x - g.alpha.y * v.y, g.alpha.x * v.y + g.alpha.y * v.x);
                    float* o = g.dst + ((b * g.rows + r) * 2) * g.ld + 2 * k;
                    *reinterpret_cast<float2*>(o) = make_float2(w.x, -w.y);         // row 2r:     Re, -Im
                    *reinterpret_cast<float2*>(o + g.ld) = make_float2(w.y, w.x);   // row 2r + 1: Im,  Re
                } else {
                    *reinterpret_cast<float2*>(g.dst + (b * g.rows + r) * g.ld + 2 * k) = v;
                }
            }
        }
        __syncthreads();
    }
}

// C *= beta (complex), through the tables.
__global__ void __launch_bounds__(256) scale_output_kernel(float2* c, const int64_t* c_b, const int64_t* c_m,
                                                           const int64_t* c_n, int64_t M, int64_t N, int64_t B, float2 beta) {
    const int64_t total = M * N * B, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int64_t m = idx % M, rest = idx / M, n = rest % N, b = rest / N;
        float2* p = c + c_b[b] + c_m[m] + c_n[n];
        const float2 o = *p;
        *p = make_float2(beta.x * o.x - beta.y * o.y, beta.x * o.y + beta.y * o.x);
    }
}

// B can serve as B' in place when its contracted modes follow one another from unit stride on, nothing
// is conjugated, and every other stride keeps the doubled (float) strides 16-byte aligned.
bool b_is_real_view(const ContractProblem& p) {
    if (p.conj_b || p.k.empty()) return false;
    int64_t run = 1;
    for (const Mode& m : p.k) {
        if (m.s[1] != run) return false;
        run *= m.extent;
    }
    if ((uintptr_t)p.b % 16 != 0 || p.n.size() > 2 || p.batch.size() > 1) return false;
    for (const Mode& m : p.n)
        if (m.extent > 1 && (m.s[1] <= 0 || (2 * m.s[1]) % 4 != 0)) return false;
    for (const Mode& m : p.batch)
        if (m.extent > 1 && (m.s[1] <= 0 || (2 * m.s[1]) % 4 != 0)) return false;
    return true;
}

}  // namespace

// Bytes that a patch or a tile moves per element of 8 where its lanes run along `g` in tensor t: a sector each unless neighbours
// share one.
static double lane_bytes(const std::vector<Mode>& g, int t) {
    if (g.empty() || std::llabs(g[0].s[t]) != 1) return 32;
    return std::max(8.0, 32.0 / (double)g[0].extent);
}
static double gather_bytes(const ContractProblem& p, const std::vector<Mode>& free, int t) {
    return std::min(lane_bytes(free, t), lane_bytes(p.k, t));
}

// What tiles of 128 columns (the second operand's rows) compute over what they keep, where B serves in place with two modes.
static double in_place_padding(const ContractProblem& p) {
    if (p.n.size() != 2) return 1;
    const int64_t e1 = p.n[0].extent;
    return e1 < 128 && 128 % e1 == 0 ? 1 : (double)((e1 + 127) / 128 * 128) / (double)e1;
}
// In place, unless the tiles' padding costs more than the copy: some 8 operations at 100 TFLOP/s per padded element and row
// against 24 bytes at 5 TB/s (162 rows, K = 16200, 20 of every 128 columns kept: 430 us in place, 95 and a copy of 35; 40 rows,
// K = 32, 40 of 128 columns: 66 us a call in place, 49 copied).  One contracted mode is read in place as it always was:
// short, and bound by the output.
static bool second_in_place(const ContractProblem& p) {
    if (!b_is_real_view(p) || !env_int("TFB_C32_B_IN_PLACE", 1)) return false;
    return p.k.size() == 1 || (in_place_padding(p) - 1) * (double)p.M() < 64;
}

// Rows in the first operand's order or the output's, K in the first operand's or the second's: whatever moves the fewest bytes.
// The first operand is gathered (and its 2 x 2 blocks written) in any order, so rows by the output cost nothing where the gather's
// lanes keep a unit stride - a tile whose rows follow the operand instead stores every element to a sector of its own (the
// outer-product node of a network with extents 79, 66, 94, 68, 86, 96, 72, 11352 x 6912 x 136 floats: 727 us by the operand's
// order, 183 by the output's) - and K by the second operand spares the copy of that (130 us
// for 5427 x 5760 elements) unless it scatters the gather of a larger first one ('efdab,fdce->abfc', 2016 x 4428 against 506 x 4428 in
// eight products: set-up 1096 us by the second operand's order, 504 by the first's).
static double embedding_bytes(const ContractProblem& p) {
    const double M = (double)p.M(), N = (double)p.N(), K = (double)p.K();
    const double second = second_in_place(p) ? 0.4 * (in_place_padding(p) - 1) * M : gather_bytes(p, p.n, 1) + 8;
    return M * K * (gather_bytes(p, p.m, 0) + 16) + N * K * second + M * N * lane_bytes(p.m, 2);
}
static ContractProblem embedding_order(const ContractProblem& p) {
    auto by = [](std::vector<Mode>& g, int t) {
        for (const Mode& m : g)
            if (m.s[t] == 0) return;
        std::stable_sort(g.begin(), g.end(), [t](const Mode& x, const Mode& y) { return std::llabs(x.s[t]) < std::llabs(y.s[t]); });
    };
    ContractProblem best;
    double least = 0;
    for (int order = 0; order < 4; ++order) {
        ContractProblem q = p;
        by(q.m, order & 1 ? 0 : 2);
        by(q.k, order & 2 ? 0 : 1);
        const double bytes = embedding_bytes(q);
        if (order == 0 || bytes < 0.95 * least) {
            least = bytes;
            best = q;
        }
    }
    return best;
}

static tfb_status embedded_product(tfb_ctx* ctx, const ContractProblem& p, bool* declined) {
    *declined = true;
    if (p.dtype != TFB_C32 || env_int("TFB_NO_TCGEN05", 0)) return TFB_OK;
    const int64_t M = p.M(), N = p.N(), K = p.K(), B = p.B();
    if (2 * M < 32 || N < 32 || K < 4) return TFB_OK;
    const int64_t ld = (2 * K + 3) / 4 * 4;  // rows of the packed operands start on 16-byte boundaries
    if (2 * M * ld * B > (int64_t)1 << 40 || N * ld * B > (int64_t)1 << 40) return TFB_OK;
    std::shared_ptr<ContractTables> t;
    TFB_TRY(get_tables(ctx, p, &t));
    ContractArgs ca;
    fill_args(p, t.get(), &ca);

    const bool b_in_place = second_in_place(p);
    const size_t a_floats = (size_t)(2 * M * ld * B), b_floats = b_in_place ? 0 : (size_t)(N * ld * B);
    const size_t tab_entries = (size_t)(2 * M + N + B);
    PoolBlock ws;
    TFB_TRY(ws.alloc(ctx, (a_floats + b_floats) * sizeof(float) + tab_entries * sizeof(int64_t) + 256));
    float* a_real = (float*)ws.ptr;
    float* b_real = a_real + a_floats;
    int64_t* tab_m = (int64_t*)(((uintptr_t)(b_real + b_floats) + 15) & ~(uintptr_t)15);
    int64_t* tab_n = tab_m + 2 * M;
    int64_t* tab_b = tab_n + N;

    const int64_t for_tables = (std::max<int64_t>(std::max<int64_t>(2 * M, N), B) + 255) / 256;
    auto patches = [&](int64_t rows) { return ((rows + 31) / 32) * ((K + 31) / 32) * B; };
    const float2 alpha = make_float2((float)p.alpha.re, (float)p.alpha.im);
    const EmbedArgs first{(const float2*)p.a, t->a_m, t->a_k, t->a_b, M, K, B, ld, ca.a_kfast, p.conj_a, 1, alpha, a_real};
    const EmbedArgs second{(const float2*)p.b, t->b_n, t->b_k, t->b_b, N, K, B, ld, ca.b_kfast, p.conj_b, 0, make_float2(1.f, 0.f), b_real};
    const RealTables tables{t->c_m, t->c_n, t->c_b, M, N, B, tab_m, tab_n, tab_b};
    auto scattered = [&](const std::vector<Mode>& g, int t, int64_t rows) {
        return gather_bytes(p, g, t) > 16 && 8.0 * (double)rows * (double)K * (double)B > 64e6;
    };
    double beta = p.beta.re;
    if (p.beta.im != 0) {
        const int64_t blocks = (M * N * B + 255) / 256;
        LaunchScope ls(ctx, "scale");
        scale_output_kernel<<<(unsigned)std::min<int64_t>(blocks, (int64_t)ctx->sm_count * 32), 256, 0, ctx->stream>>>(
            (float2*)p.c, t->c_b, t->c_m, t->c_n, M, N, B, make_float2((float)p.beta.re, (float)p.beta.im));
        TFB_CUDA(cudaGetLastError());
        beta = 1.0;
    }

    // The set-up kernels, which contract_tcgen05 has run once it knows whether the product runs on split operands.
    auto pass = [&](const Gate& gate, bool scatters, int64_t blocks, int job0, unsigned jobs) -> tfb_status {
        LaunchScope ls(ctx, "pack_planes");
        const dim3 grid((unsigned)std::min<int64_t>(blocks, (int64_t)ctx->sm_count * (gate.word ? 8 : 16)), jobs);
        TFB_CUDA(scatters ? launch_overlapped(ctx, embed_setup_kernel<true>, grid, dim3(256), 0, 0u, first, second, tables, job0, gate)
                          : launch_overlapped(ctx, embed_setup_kernel<false>, grid, dim3(256), 0, 0u, first, second, tables, job0, gate));
        return TFB_OK;
    };
    const bool a_scatters = scattered(p.m, 0, M), b_scatters = !b_in_place && scattered(p.n, 1, N);
    const std::function<tfb_status(const Gate&)> set_up = [&](const Gate& gate) -> tfb_status {
        if (b_in_place || a_scatters || b_scatters) {
            TFB_TRY(pass(gate, a_scatters, std::max(for_tables, patches(M)), 0, 2));
            if (!b_in_place) TFB_TRY(pass(gate, b_scatters, patches(N), 2, 1));
        } else {
            TFB_TRY(pass(gate, false, std::max({for_tables, patches(M), patches(N)}), 0, 3));
        }
        return TFB_OK;
    };
    // The real product: A' [B][2M][ld] K-major, B' [B][N][ld] K-major (or B itself), C through the tables.
    ContractProblem q;
    q.dtype = TFB_F32;
    q.a = a_real;
    q.b = b_in_place ? p.b : (const void*)b_real;
    q.c = p.c;
    q.alpha = Scalar{1.0, 0.0};
    q.beta = Scalar{beta, 0.0};
    if (b_in_place) {
        if (B > 1) q.batch.push_back(Mode{B, {2 * M * ld, 2 * p.batch[0].s[1], 0}});
        for (const Mode& m : p.n) q.n.push_back(Mode{m.extent, {0, 2 * m.s[1], 0}});
    } else {
        if (B > 1) q.batch.push_back(Mode{B, {2 * M * ld, N * ld, 0}});
        q.n.push_back(Mode{N, {0, ld, 0}});
    }
    q.m.push_back(Mode{2 * M, {ld, 0, 0}});
    q.k.push_back(Mode{2 * K, {1, 1, 0}});
    const int64_t* c_tables[3] = {tab_b, tab_m, tab_n};
    // What the set-up kernels would write, split into 16-bit halves instead.  Scattered operands keep the kernels that are made
    // for them.
    SplitProduct split{};
    split.a = SplitOperand{p.a, t->a_m, t->a_k, t->a_b, M, K, B, SplitOperand::Embedded, ca.a_kfast, p.conj_a, alpha,
                           one_step(p.m, 0), one_step(p.k, 0), common_step(p.batch, 0)};
    split.b = SplitOperand{p.b, t->b_n, t->b_k, t->b_b, N, K, B, SplitOperand::Parts, ca.b_kfast, p.conj_b, make_float2(1.f, 0.f),
                           one_step(p.n, 1), one_step(p.k, 1), common_step(p.batch, 1)};
    split.M = 2 * M;
    split.N = N;
    split.K = 2 * K;
    split.B = B;
    split.c = p.c;
    split.complex_b = t->c_b;
    split.complex_m = t->c_m;
    split.complex_n = t->c_n;
    split.complex_rows = true;
    if (!p.n.empty() && p.n.size() <= 2 && p.n[0].extent < INT32_MAX) {
        split.cn_e1 = p.n.size() == 2 ? (int)p.n[0].extent : INT32_MAX;
        split.cn_s1 = 2 * p.n[0].s[2];
        split.cn_s2 = p.n.size() == 2 ? 2 * p.n[1].s[2] : 0;
    }
    split.alpha = 1.f;
    split.beta = (float)beta;
    split.m_modes = &p.m;
    split.n_modes = &p.n;
    split.c_scale = 2;
    split.cols_fast = !p.n.empty() && std::llabs(p.n[0].s[2]) == 1;
    const bool pays = !a_scatters && !b_scatters && split_pays(2 * M, N, 2 * K, B, b_in_place ? 16.0 * (double)N * (double)K * (double)B : 0);
    bool d = false;
    TFB_TRY(contract_tcgen05(ctx, q, &d, c_tables, &p.n, 2, &p.m, &p.batch, pays ? &split : nullptr, &set_up));
    if (d) return fail(TFB_ERR_DEVICE, "internal: the embedded real product was declined by the tensor-core kernel");
    *declined = false;
    return TFB_OK;
}

// Floats the set-up kernels of embedded_product write: the 2 x 2 embedding of the first operand
// (2M x 2K), and a K-major copy of the second (N x 2K) unless it serves in place.
static double setup_floats(const ContractProblem& p) {
    const double k2 = 2.0 * (double)p.K() * (double)p.B();
    return 2.0 * (double)p.M() * k2 + (second_in_place(p) ? 0.0 : (double)p.N() * k2);
}

tfb_status contract_c32_embedded(tfb_ctx* ctx, const ContractProblem& p, bool* declined) {
    if (!p.mul) {
        // The embedded operand should be the small one: a tall first operand against a short second
        // one (M >> N) would spend more time being embedded than the product takes.
        if (env_int("TFB_C32_EXCHANGE", 1)) {
            const ContractProblem q = embedding_order(exchange_roles(p));
            if (setup_floats(q) < 0.6 * setup_floats(embedding_order(p))) return embedded_product(ctx, q, declined);
        }
        return embedded_product(ctx, embedding_order(p), declined);
    }
    // A fused multiplier is a complex product per element, and the real embedding holds the two
    // parts of an element in different rows: the product runs unfused and C is multiplied in
    // place afterwards (no intermediate tensor).  With a beta term the exact kernel takes it.
    *declined = true;
    if (!p.beta.is_zero()) return TFB_OK;
    ContractProblem q = p;
    q.mul = nullptr;
    q.conj_mul = false;
    TFB_TRY(embedded_product(ctx, embedding_order(q), declined));
    if (*declined) return TFB_OK;
    std::vector<Mode> all;
    for (auto* g : {&p.m, &p.n, &p.batch})
        for (auto& m : *g) all.push_back(Mode{m.extent, {m.s[2], m.s[3], m.s[2]}});
    sort_and_fuse(all, 2, 3);
    LoopNest nest;
    TFB_TRY(make_nest(all, &nest));
    return launch_elementwise_mul(ctx, p.dtype, nest, p.c, p.mul, p.c, Scalar{1.0, 0.0}, Scalar{0.0, 0.0}, false, p.conj_mul);
}

}  // namespace tfb
