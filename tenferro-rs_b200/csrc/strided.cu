// Bandwidth-bound strided kernels: permute, element-wise product, reduce, scale.
// They implement `PrimDescriptor::{Permute, ElementwiseMul, Reduce}` and the alpha/beta
// contract of `TensorPrims::execute` (tenferro-prims/src/lib.rs:170-202, 241-244, 300-320)
// on arbitrary signed element strides.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.h"
#include "ptx_sm100.cuh"
#include "scalar_ops.cuh"

namespace tfb {

// ------------------------------------------------------------------ index helpers
__device__ __forceinline__ void divmod(int64_t idx, int64_t e, int64_t& q, int64_t& r) {
    if ((uint64_t)idx <= 0xffffffffull && (uint64_t)e <= 0xffffffffull) {
        uint32_t a = (uint32_t)idx, b = (uint32_t)e;
        uint32_t qq = a / b;
        q = qq;
        r = a - qq * b;
    } else {
        q = idx / e;
        r = idx - q * e;
    }
}

// Decompose a linear index over modes [first, nest.rank) (mode `first` fastest) into offsets.
template <int NT>
__device__ __forceinline__ void decompose(const LoopNest& nest, int first, int64_t idx, int64_t (&off)[NT]) {
#pragma unroll
    for (int t = 0; t < NT; ++t) off[t] = 0;
    for (int d = first; d < nest.rank; ++d) {
        int64_t q, r;
        divmod(idx, nest.extent[d], q, r);
#pragma unroll
        for (int t = 0; t < NT; ++t) off[t] += r * nest.stride[t][d];
        idx = q;
    }
}

// Division by an invariant 32-bit divisor as a multiplication and a shift (Granlund and Montgomery,
// "Division by invariant integers using multiplication", PLDI 1994), for numerators below 2^31.
struct FastDiv {
    uint32_t d, mul, shift;
    static FastDiv of(uint32_t d) {
        uint32_t shift = 0;
        while ((1ull << shift) < d) ++shift;
        return FastDiv{d, (uint32_t)((((1ull << shift) - d) << 32) / d + 1), shift};
    }
    __device__ __forceinline__ uint32_t quotient(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};
// A loop nest of fewer than 2^31 elements: no hardware division per element and mode.
struct Nest32 {
    int rank;
    FastDiv div[kMaxRank];
    int64_t stride[3][kMaxRank];
    int64_t total;
    explicit Nest32(const LoopNest& n) : rank(n.rank), total(n.total) {
        for (int d = 0; d < kMaxRank; ++d) {
            div[d] = FastDiv::of(d < n.rank ? (uint32_t)n.extent[d] : 1u);
            for (int t = 0; t < 3; ++t) stride[t][d] = n.stride[t][d];
        }
    }
    static bool fits(const LoopNest& n) { return n.total > 0 && n.total < ((int64_t)1 << 31); }
};
template <int NT>
__device__ __forceinline__ void decompose(const Nest32& nest, int first, int64_t idx, int64_t (&off)[NT]) {
#pragma unroll
    for (int t = 0; t < NT; ++t) off[t] = 0;
    uint32_t i = (uint32_t)idx;
    for (int d = first; d < nest.rank; ++d) {
        uint32_t r = i;
        if (d + 1 < nest.rank) {
            const uint32_t q = nest.div[d].quotient(i);
            r = i - q * nest.div[d].d;
            i = q;
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) off[t] += r * nest.stride[t][d];
    }
}
__device__ __forceinline__ void divide_inner(const LoopNest& n, int64_t v, int64_t u, int64_t& q, int64_t& r) {
    divmod(u, n.extent[0] / v, q, r);
}
// (for v > 1 the host has made div[0] a divider by units of v elements)
__device__ __forceinline__ void divide_inner(const Nest32& n, int64_t, int64_t u, int64_t& q, int64_t& r) {
    const uint32_t qq = n.div[0].quotient((uint32_t)u);
    q = qq;
    r = (uint32_t)u - qq * n.div[0].d;
}

// ------------------------------------------------------------------ permute
// General path: linear over the nest in OUTPUT order (mode 0 = output's fastest), so writes
// coalesce; reads are whatever the input strides give.
template <typename T, typename N>
__global__ void __launch_bounds__(256) permute_generic_kernel(N nest, const T* in, T* out,
                                                              EpilogueArgs<T> ep) {
    launch_begin();
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < nest.total; idx += stride) {
        int64_t off[2];
        decompose<2>(nest, 0, idx, off);
        T v = in[off[0]];
        out[off[1]] = ep.apply(v, out + off[1]);
    }
}

// Row path: mode 0 has stride 1 in both tensors.  V elements per thread move as one 16-byte
// access when `vec` holds (alignment checked on the host).
template <typename T, int V, typename N>
__global__ void __launch_bounds__(256) permute_rows_kernel(N nest, const T* in, T* out,
                                                           EpilogueArgs<T> ep) {
    launch_begin();
    // One "unit" = V consecutive elements of mode 0.
    const int64_t units = nest.total / V;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ep.plain) {
        // Pure copy: four units per thread, all loads issued before the first store.
        for (; u + 3 * stride < units; u += 4 * stride) {
            Pack<T, V> p[4];
            T* dst[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int64_t q, r;
                divide_inner(nest, V, u + k * stride, q, r);
                int64_t off[2];
                decompose<2>(nest, 1, q, off);
                p[k] = *reinterpret_cast<const Pack<T, V>*>(in + off[0] + r * V);
                dst[k] = out + off[1] + r * V;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) *reinterpret_cast<Pack<T, V>*>(dst[k]) = p[k];
        }
    }
    for (; u < units; u += stride) {
        int64_t q, r;
        divide_inner(nest, V, u, q, r);
        int64_t off[2];
        decompose<2>(nest, 1, q, off);
        const T* src = in + off[0] + r * V;
        T* dst = out + off[1] + r * V;
        Pack<T, V> p = *reinterpret_cast<const Pack<T, V>*>(src);
        if (ep.plain) {
            *reinterpret_cast<Pack<T, V>*>(dst) = p;
        } else {
            Pack<T, V> o;
            if (ep.read_out) o = *reinterpret_cast<const Pack<T, V>*>(dst);
#pragma unroll
            for (int i = 0; i < V; ++i) o.v[i] = ep.apply(p.v[i], &o.v[i]);
            *reinterpret_cast<Pack<T, V>*>(dst) = o;
        }
    }
}

// CTAs of a kernel whose threads take up to four units each: one unit while the chip has room for all of them at
// once (8 CTAs an SM), since a thread's four follow one another where there are few (57 x 128 complex double copied:
// 5.8 us with four, 4.4 with one).
static unsigned grid_of_four(int64_t units, int sms, int most) {
    const int64_t one = (units + 255) / 256, room = (int64_t)sms * 8;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(std::max<int64_t>(std::min(one, room), (units + 1023) / 1024), (int64_t)sms * most));
}

// Tiled transpose path: mode 0 is the input's stride-1 mode ("i"), mode 1 the output's
// stride-1 mode ("j").  A TILE x TILE patch goes through shared memory so that both the
// reads (along i) and the writes (along j) are full 128-byte lines.  Tiles run eight along i, then along j: with odd
// extents neighbours share sectors in both directions, and a neighbour along j that comes 100 MB later
// finds its half-written sectors gone from L2 (229273 x 369 complex double transposed: 620 -> 454 us).
template <typename T>
struct TileOf {
    static constexpr int value = sizeof(T) >= 16 ? 32 : 64;  // keeps the patch under 48 KB
};
template <typename T>
__global__ void __launch_bounds__(256) permute_tiled_kernel(LoopNest nest, const T* in, T* out,
                                                            EpilogueArgs<T> ep, int64_t tiles_i, int64_t tiles_j,
                                                            int64_t n_tiles, int64_t strip, int64_t strips) {
    launch_begin();
    constexpr int kTile = TileOf<T>::value;
    constexpr int kStep = 256 / kTile;
    // Odd pitch: a column walk hits distinct banks.
    __shared__ T tile[kTile][kTile + 1];
    const int tx = threadIdx.x % kTile, ty = threadIdx.x / kTile;
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        int64_t q, strip_i, ti, tj, rest;
        if constexpr (sizeof(T) == 4) {  // nothing gained by strips (27757 x 374: 18.3 us without, 19.6 with)
            divmod(t, tiles_i, q, ti);
            divmod(q, tiles_j, rest, tj);
        } else {
            divmod(t, strip, q, strip_i);
            divmod(q, tiles_j, q, tj);
            divmod(q, strips, rest, ti);
            ti = ti * strip + strip_i;
            if (ti >= tiles_i) continue;
        }
        int64_t off[2];
        decompose<2>(nest, 2, rest, off);
        const int64_t i0 = ti * kTile, j0 = tj * kTile;
        const int64_t ni = min((int64_t)kTile, nest.extent[0] - i0), nj = min((int64_t)kTile, nest.extent[1] - j0);
        const T* src = in + off[0] + i0 * nest.stride[0][0] + j0 * nest.stride[0][1];
        T* dst = out + off[1] + i0 * nest.stride[1][0] + j0 * nest.stride[1][1];
        const int64_t s_in_j = nest.stride[0][1], s_out_i = nest.stride[1][0];
        // Load: threads along i (input stride 1).
        if (tx < ni) {
#pragma unroll 4
            for (int j = ty; j < nj; j += kStep) tile[j][tx] = src[tx + j * s_in_j];
        }
        __syncthreads();
        // Store: threads along j (output stride 1).
        if (tx < nj) {
#pragma unroll 4
            for (int i = ty; i < ni; i += kStep) {
                T* p = dst + tx + i * s_out_i;
                *p = ep.apply(tile[tx][i], p);
            }
        }
        __syncthreads();
    }
}

// Tile path, for any order of any number of modes.  The modes are split into a run R that has unit stride in both
// tensors (usually empty), a group I that is dense, or nearly, where the input is walked, a group J likewise for
// the output, and the rest.  A tile is a patch of (R x) I x J through shared memory: it is read with
// neighbouring threads along (R, I) and written with neighbouring threads along (R, J), so both
// sides move whole sectors even where single extents are short.  Offsets inside a tile come from four tables
// in shared memory, made once per tile; an element's place in its table is a multiplication and a shift.
// All loads of a thread are issued before the first is used.  Neighbouring tiles in both directions run close in
// time, since with odd extents they share sectors.
// Bound by HBM for large tensors.  14 x 89 x 15 x 10 x 149 f64 in the order 4,2,3,1,0: 481 -> 110 us (generic
// kernel), 27 x 9 x 68 x 24 x 84 f64 in 4,1,3,0,2: 227 -> 163 (square tiles of two modes).  Some 35 instructions per
// element keep f32 at 2 TB/s.
constexpr int kSide = 256;  // longest side of a tile, (R, I) or (R, J)
template <typename T>
constexpr int kPatch = sizeof(T) >= 16 ? 2048 : 4096;  // elements of a tile

struct TileGroup {
    int rank = 0;
    FastDiv div[kMaxRank];
    int32_t in[kMaxRank], out[kMaxRank];
    uint32_t total = 1, width = 1, tiles = 1;
    __device__ __forceinline__ void offsets(uint32_t idx, int32_t& o_in, int32_t& o_out) const {
        o_in = o_out = 0;
        for (int d = 0; d < rank; ++d) {
            const uint32_t q = div[d].quotient(idx), r = idx - q * div[d].d;
            o_in += (int32_t)r * in[d];
            o_out += (int32_t)r * out[d];
            idx = q;
        }
    }
};
struct TilePlan {
    TileGroup I, J;
    FastDiv run;                   // R
    FastDiv side_i[2], side_j[2];  // R * width of a whole and of the last tile
    LoopNest rest;
    int64_t n_tiles;  // in strips along I, the last one filled up
    uint32_t strip, strips;
};

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 3) permute_tile_kernel(const __grid_constant__ TilePlan p, const T* in, T* out,
                                                           EpilogueArgs<T> ep) {
    launch_begin();
    constexpr int L = kPatch<T> / 256;
    __shared__ T patch[kPatch<T> + kSide];
    __shared__ int32_t in_i[kSide], in_j[kSide], out_i[kSide], out_j[kSide];
    const int tid = threadIdx.x;
    const uint32_t R = p.run.d;
    for (int64_t t = blockIdx.x; t < p.n_tiles; t += gridDim.x) {
        int64_t q, tj, s, strip_i, rest;
        divmod(t, p.strip, q, strip_i);
        divmod(q, p.J.tiles, q, tj);
        divmod(q, p.strips, rest, s);
        const uint32_t ti = (uint32_t)s * p.strip + (uint32_t)strip_i;
        if (ti >= p.I.tiles) continue;
        int64_t off[2];
        decompose<2>(p.rest, 0, rest, off);
        const T* src = in + off[0];
        T* dst = out + off[1];
        const uint32_t i0 = ti * p.I.width, j0 = (uint32_t)tj * p.J.width;
        const uint32_t wi = min(p.I.width, p.I.total - i0), wj = min(p.J.width, p.J.total - j0);
        const FastDiv di = p.side_i[ti + 1 == p.I.tiles], dj = p.side_j[tj + 1 == p.J.tiles];
        const uint32_t pitch = (R * wj) | 1, count = R * wi * wj;
        if (tid < (int)di.d) {
            const uint32_t i = p.run.quotient(tid), r = tid - i * R;
            int32_t a, b;
            p.I.offsets(i0 + i, a, b);
            in_i[tid] = a + (int32_t)r;
            if (r == 0) out_i[i] = b;
        }
        if (tid < (int)dj.d) {
            const uint32_t j = p.run.quotient(tid), r = tid - j * R;
            int32_t a, b;
            p.J.offsets(j0 + j, a, b);
            out_j[tid] = b + (int32_t)r;
            if (r == 0) in_j[j] = a;
        }
        __syncthreads();
        T v[L];
        uint32_t at[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const uint32_t e = tid + 256 * k;
            if (e >= count) continue;
            const uint32_t j = di.quotient(e), ir = e - j * di.d;
            v[k] = src[(int64_t)in_i[ir] + in_j[j]];
            const uint32_t i = R == 1 ? ir : p.run.quotient(ir);
            at[k] = i * pitch + j * R + (ir - i * R);
        }
#pragma unroll
        for (int k = 0; k < L; ++k)
            if (tid + 256 * k < count) patch[at[k]] = v[k];
        __syncthreads();
        if (ep.read_out) {
            // all of a thread's outputs are on their way before the first store
#pragma unroll
            for (int k = 0; k < L; ++k) {
                const uint32_t e = tid + 256 * k;
                if (e >= count) continue;
                const uint32_t i = dj.quotient(e), jr = e - i * dj.d;
                v[k] = dst[(int64_t)out_j[jr] + out_i[i]];
            }
        }
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const uint32_t e = tid + 256 * k;
            if (e >= count) continue;
            const uint32_t i = dj.quotient(e), jr = e - i * dj.d;
            dst[(int64_t)out_j[jr] + out_i[i]] = ep.apply(patch[i * pitch + jr], &v[k]);
        }
        __syncthreads();
    }
}

// Fits the tile path to a nest in output order (mode 0 fastest); false where another path is the better one.
template <typename T>
static bool plan_tiles(const LoopNest& n, int sms, TilePlan* p) {
    if (n.rank < 2 || n.total >= ((int64_t)1 << 31) || n.stride[1][0] != 1) return false;
    // Tiles for less than six tenths of the SMs: a tile's latency is longer than that of the one element a thread moves
    // on the other paths (us there and in tiles: 54432 f64 4.8, 7.2; 349272 f32 6.3, 9.2; 599760 f32 10.3, 8.4; 425776
    // complex double 8.8, 7.0).
    if (n.total * 10 < (int64_t)sms * 6 * kPatch<T>) return false;
    auto mag = [](int64_t v) { return v < 0 ? -v : v; };
    int im = -1;
    for (int d = 0; d < n.rank; ++d)
        if (n.stride[0][d] == 1) im = d;
    if (im < 0) return false;
    bool taken[kMaxRank] = {};
    int64_t R = 1;
    if (im == 0) {
        R = n.extent[0];
        taken[0] = true;
    }
    // the free mode nearest to memory in tensor t, broadcast modes last
    auto nearest = [&](int t) {
        int best = -1;
        for (int d = 0; d < n.rank; ++d) {
            if (taken[d] || n.stride[t][d] == 0) continue;
            if (best < 0 || mag(n.stride[t][d]) < mag(n.stride[t][best])) best = d;
        }
        return best;
    };
    std::vector<int> gi, gj;
    int64_t ni = 1, nj = 1;
    if (nearest(0) < 0 || nearest(0) == nearest(1)) return false;  // a run and then the same order: rows
    const int64_t want = std::max<int64_t>(1, 64 / R);
    while (ni < want || nj < want) {
        const bool grow_i = ni < want && (ni <= nj || nj >= want);
        const int d = nearest(grow_i ? 0 : 1);
        if (d < 0) break;
        taken[d] = true;
        (grow_i ? gi : gj).push_back(d);
        (grow_i ? ni : nj) *= n.extent[d];
    }
    if (gi.empty() || gj.empty()) return false;
    auto fill = [&](const std::vector<int>& g, TileGroup* o) {
        double span[2] = {0, 0};
        for (int d : g) {
            o->div[o->rank] = FastDiv::of((uint32_t)n.extent[d]);
            for (int t = 0; t < 2; ++t) span[t] += (double)(n.extent[d] - 1) * (double)mag(n.stride[t][d]);
            if (span[0] > 1e9 || span[1] > 1e9) return false;
            o->in[o->rank] = (int32_t)n.stride[0][d];
            o->out[o->rank++] = (int32_t)n.stride[1][d];
            o->total *= (uint32_t)n.extent[d];
        }
        return true;
    };
    *p = TilePlan{};
    if (!fill(gi, &p->I) || !fill(gj, &p->J)) return false;
    // 64 on each side, more where the other side is short, in equal parts
    auto width = [&](int64_t total, int64_t most) {
        const int64_t w = std::max<int64_t>(1, std::min<int64_t>(most, kSide / R)), parts = (total + w - 1) / w;
        return (total + parts - 1) / parts;
    };
    const int64_t patch = kPatch<T>, half = sizeof(T) >= 16 ? 45 : 64;
    int64_t wi = width(ni, half / R);
    const int64_t wj = width(nj, patch / (R * wi));
    wi = width(ni, patch / (R * wj));
    p->I.width = (uint32_t)wi;
    p->J.width = (uint32_t)wj;
    p->I.tiles = (uint32_t)((ni + wi - 1) / wi);
    p->J.tiles = (uint32_t)((nj + wj - 1) / wj);
    p->run = FastDiv::of((uint32_t)R);
    p->side_i[0] = FastDiv::of((uint32_t)(R * wi));
    p->side_i[1] = FastDiv::of((uint32_t)(R * (ni - (p->I.tiles - 1) * wi)));
    p->side_j[0] = FastDiv::of((uint32_t)(R * wj));
    p->side_j[1] = FastDiv::of((uint32_t)(R * (nj - (p->J.tiles - 1) * wj)));
    LoopNest& rest = p->rest;
    rest.rank = 0;
    rest.total = 1;
    for (int d = 0; d < n.rank; ++d) {
        if (taken[d]) continue;
        rest.extent[rest.rank] = n.extent[d];
        for (int t = 0; t < 3; ++t) rest.stride[t][rest.rank] = n.stride[t][d];
        rest.total *= n.extent[d];
        ++rest.rank;
    }
    p->strips = (p->I.tiles + 7) / 8;
    p->strip = (p->I.tiles + p->strips - 1) / p->strips;
    p->n_tiles = (int64_t)p->strip * p->strips * p->J.tiles * rest.total;
    return true;
}

// Vector form of the tiled transpose of two modes (0: the input's unit stride, 1: the output's) for 4- and 8-byte elements: 16-byte loads along the
// input's unit stride, 16-byte stores along the output's, every load of a thread issued before
// the first use (16 KB in flight per CTA; MINB CTAs per SM).  Needs both sides 16-byte aligned.
template <typename T, int V, int MINB>
__global__ void __launch_bounds__(256, MINB) permute_tiled_vec_kernel(LoopNest nest, const T* in, T* out,
                                                                EpilogueArgs<T> ep, int64_t tiles_i, int64_t tiles_j,
                                                                int64_t n_tiles) {
    launch_begin();
    constexpr int TILE = 64, VPR = TILE / V, LOADS = TILE * TILE / V / 256;
    __shared__ T tile[TILE][TILE + 1];  // tile[i][j]
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        int64_t q, ti, tj, rest;
        divmod(t, tiles_i, q, ti);
        divmod(q, tiles_j, rest, tj);
        int64_t off[2];
        decompose<2>(nest, 2, rest, off);
        const int64_t i0 = ti * TILE, j0 = tj * TILE;
        const int ni = (int)min((int64_t)TILE, nest.extent[0] - i0), nj = (int)min((int64_t)TILE, nest.extent[1] - j0);
        const T* src = in + off[0] + i0 * nest.stride[0][0] + j0 * nest.stride[0][1];
        T* dst = out + off[1] + i0 * nest.stride[1][0] + j0 * nest.stride[1][1];
        const int64_t s_in_j = nest.stride[0][1], s_out_i = nest.stride[1][0];
        Pack<T, V> v[LOADS];
#pragma unroll
        for (int r = 0; r < LOADS; ++r) {
            const int c = threadIdx.x + 256 * r, i = (c % VPR) * V, j = c / VPR;
            if (i < ni && j < nj) v[r] = *reinterpret_cast<const Pack<T, V>*>(src + i + j * s_in_j);
        }
#pragma unroll
        for (int r = 0; r < LOADS; ++r) {
            const int c = threadIdx.x + 256 * r, i = (c % VPR) * V, j = c / VPR;
            if (i < ni && j < nj) {
#pragma unroll
                for (int e = 0; e < V; ++e) tile[i + e][j] = v[r].v[e];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < LOADS; ++r) {
            const int c = threadIdx.x + 256 * r, j = (c % VPR) * V, i = c / VPR;
            if (j < nj && i < ni) {
                Pack<T, V>* p = reinterpret_cast<Pack<T, V>*>(dst + j + i * s_out_i);
                Pack<T, V> o;
                if (ep.read_out) o = *p;
#pragma unroll
                for (int e = 0; e < V; ++e) o.v[e] = ep.apply(tile[i][j + e], &o.v[e]);
                *p = o;
            }
        }
        __syncthreads();
    }
}

template <typename T>
static tfb_status permute_typed(tfb_ctx* ctx, const LoopNest& nest_out_order, const void* in, void* out, Scalar alpha,
                                Scalar beta, bool conj) {
    EpilogueArgs<T> ep = EpilogueArgs<T>::make(alpha, beta, conj);
    LoopNest nest = nest_out_order;
    if (nest.total == 0) return TFB_OK;
    const int sms = ctx->sm_count;
    TilePlan tiles;
    auto run_tiles = [&]() -> tfb_status {
        const unsigned grid = (unsigned)std::min<int64_t>(tiles.n_tiles, (int64_t)sms * 32);
        LaunchScope ls(ctx, "permute_tile");
        launch_overlapped(ctx, permute_tile_kernel<T>, dim3(grid), dim3(256), 0, 0u, tiles, (const T*)in, (T*)out, ep);
        TFB_CUDA(cudaGetLastError());
        return TFB_OK;
    };
    // Row path: both tensors walk mode 0.
    if (nest.rank >= 1 && nest.stride[0][0] == 1 && nest.stride[1][0] == 1) {
        constexpr int VMAX = 16 / sizeof(T) > 0 ? 16 / sizeof(T) : 1;
        bool vec = VMAX > 1 && nest.extent[0] % VMAX == 0 && ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0);
        for (int d = 1; d < nest.rank && vec; ++d)
            vec = nest.stride[0][d] % VMAX == 0 && nest.stride[1][d] % VMAX == 0;
        // Short rows of 8- and 16-byte elements whose neighbours in the output lie a megabyte or more apart in the input
        // reach HBM as single sectors: there the tile path, which gathers whole lines, is the better one (time by rows
        // over time in tiles, 16 M elements, outer modes reversed: 24 bytes f64 1.42, 56 bytes 1.13; 32 and 96 bytes complex
        // double 1.74, 1.35).  Not so with nearer neighbours (24 bytes f64 0.89, 56 bytes 0.5 to 0.9), from 72 bytes f64 on
        // (0.62), where 8-byte elements move in 16-byte accesses (0.81) and for f32 (1.1 at most, mostly 0.3 to 0.9).
        const int64_t row = nest.extent[0] * (int64_t)sizeof(T), most = sizeof(T) == 16 ? 128 : sizeof(T) == 8 && !vec ? 64 : 0;
        if (row < most && nest.rank > 1 && std::llabs(nest.stride[0][1]) * (int64_t)sizeof(T) >= (1 << 20) && plan_tiles<T>(nest, sms, &tiles))
            return run_tiles();
        const int64_t units = vec ? nest.total / VMAX : nest.total;
        const unsigned grid = grid_of_four(units, sms, 16);
        LaunchScope ls(ctx, "permute_rows");
        auto go = [&](const auto& n) {
            if (vec) launch_overlapped(ctx, permute_rows_kernel<T, VMAX, std::decay_t<decltype(n)>>, dim3(grid), dim3(256), 0, 0u, n, (const T*)in, (T*)out, ep);
            else launch_overlapped(ctx, permute_rows_kernel<T, 1, std::decay_t<decltype(n)>>, dim3(grid), dim3(256), 0, 0u, n, (const T*)in, (T*)out, ep);
        };
        if (Nest32::fits(nest)) {
            Nest32 n(nest);
            n.div[0] = FastDiv::of((uint32_t)(nest.extent[0] / (vec ? VMAX : 1)));
            go(n);
        } else {
            go(nest);
        }
        TFB_CUDA(cudaGetLastError());
        return TFB_OK;
    }
    // Two modes that fill square tiles well enough: a tile costs the same whatever is in it, but the tile path
    // above pays about three times as much per element (f64, 27 x 84 patches: 227 us square, 162 there; 87 x 22:
    // 25, 28; 171 x 125: 271, 344).  For 4-byte elements, where instructions are all that bounds it, nearer to
    // four times (20 x 299: 20.6, 25.8).
    {
        int im = -1;
        for (int d = 1; d < nest.rank && nest.stride[1][0] == 1; ++d)
            if (nest.stride[0][d] == 1) im = d;
        if (im > 0 && nest.extent[im] >= 8 && nest.extent[0] >= 8) {
            // Reorder: mode 0 <- input-fast mode, mode 1 <- output-fast mode, rest keep order.
            LoopNest r;
            r.rank = nest.rank;
            r.total = nest.total;
            int w = 0;
            auto put = [&](int d) {
                r.extent[w] = nest.extent[d];
                for (int t = 0; t < 3; ++t) r.stride[t][w] = nest.stride[t][d];
                ++w;
            };
            put(im);
            put(0);
            for (int d = 1; d < nest.rank; ++d)
                if (d != im) put(d);
            constexpr int V = 16 / sizeof(T), kTile = TileOf<T>::value;
            const int64_t ti = (r.extent[0] + kTile - 1) / kTile, tj = (r.extent[1] + kTile - 1) / kTile;
            int64_t rest = 1;
            for (int d = 2; d < r.rank; ++d) rest *= r.extent[d];
            bool vec = V > 1 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0 && r.extent[0] % V == 0 && r.extent[1] % V == 0;
            for (int d = 0; d < r.rank && vec; ++d) {
                if (d != 0 && r.stride[0][d] % V != 0) vec = false;  // every input stride but the unit one
                if (d != 1 && r.stride[1][d] % V != 0) vec = false;  // every output stride but the unit one
            }
            const double fill = (double)r.extent[0] * (double)r.extent[1] / ((double)kTile * kTile * (double)ti * (double)tj);
            if (fill < (sizeof(T) == 4 ? 0.2 : 0.3) && plan_tiles<T>(nest, sms, &tiles)) return run_tiles();
            // What has no plan (2^31 elements, spans of a group above 1e9) and puts few elements into a tile is better off
            // element by element (ms, that way and in tiles: f32 8 x 8 patches 16.6, 85.4; 12 x 12 19.4, 39.2; 15 x 15 25.1,
            // 27.1; f64 8 x 8 22.7, 142; 14 x 14 40.4, 50.5; 15 x 15 42.6, 33.2; complex double 8 x 15 47.4, 64.7).
            if (r.extent[0] * r.extent[1] >= (sizeof(T) == 4 ? 256 : 225) * ti * tj) {
                LaunchScope ls(ctx, "permute_tiled");
                if constexpr (sizeof(T) <= 8) if (vec) {
                    // CTAs per SM: each holds 16 KB of loads in flight, and HBM wants about 90 KB per SM.
                    // Six fit for 4-byte elements (40 registers); the 33 KB tiles of 8-byte elements do
                    // best at three.
                    constexpr int kOcc = sizeof(T) == 4 ? 6 : 3;
                    const unsigned grid = (unsigned)std::min<int64_t>(ti * tj * rest, (int64_t)sms * 32);
                    launch_overlapped(ctx, permute_tiled_vec_kernel<T, V, kOcc>, dim3(grid), dim3(256), 0, 0u, r, (const T*)in, (T*)out, ep, ti, tj, ti * tj * rest);
                    TFB_CUDA(cudaGetLastError());
                    return TFB_OK;
                }
                const int64_t strips = sizeof(T) == 4 ? 1 : (ti + 7) / 8, strip = (ti + strips - 1) / strips, n_tiles = strips * strip * tj * rest;
                const unsigned grid = (unsigned)std::min<int64_t>(n_tiles, (int64_t)sms * 32);
                launch_overlapped(ctx, permute_tiled_kernel<T>, dim3(grid), dim3(256), 0, 0u, r, (const T*)in, (T*)out, ep, ti, tj, n_tiles, strip, strips);
                TFB_CUDA(cudaGetLastError());
                return TFB_OK;
            }
        }
    }
    if (plan_tiles<T>(nest, sms, &tiles)) return run_tiles();
    int64_t blocks = (nest.total + 255) / 256;
    int64_t cap = (int64_t)sms * 16;
    int grid = (int)(blocks < cap ? blocks : cap);
    LaunchScope ls(ctx, "permute_generic");
    if (Nest32::fits(nest)) launch_overlapped(ctx, permute_generic_kernel<T, Nest32>, dim3(grid), dim3(256), 0, 0u, Nest32(nest), (const T*)in, (T*)out, ep);
    else launch_overlapped(ctx, permute_generic_kernel<T, LoopNest>, dim3(grid), dim3(256), 0, 0u, nest, (const T*)in, (T*)out, ep);
    TFB_CUDA(cudaGetLastError());
    return TFB_OK;
}

tfb_status launch_permute(tfb_ctx* ctx, int dtype, const LoopNest& nest, const void* in, void* out, Scalar alpha,
                          Scalar beta, bool conj) {
    DeviceGuard g(ctx->device);
    switch (dtype) {
        case TFB_F32: return permute_typed<float>(ctx, nest, in, out, alpha, beta, conj);
        case TFB_F64: return permute_typed<double>(ctx, nest, in, out, alpha, beta, conj);
        case TFB_C32: return permute_typed<float2>(ctx, nest, in, out, alpha, beta, conj);
        case TFB_C64: return permute_typed<double2>(ctx, nest, in, out, alpha, beta, conj);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

// ------------------------------------------------------------------ scale (out = beta * out)
template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(LoopNest nest, T* out, T beta, bool zero) {
    launch_begin();
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < nest.total; idx += stride) {
        int64_t off[1];
        decompose<1>(nest, 0, idx, off);
        out[off[0]] = zero ? Ops<T>::zero() : Ops<T>::mul(beta, out[off[0]]);
    }
}
template <typename T>
static tfb_status scale_typed(tfb_ctx* ctx, const LoopNest& nest, void* out, Scalar beta) {
    if (nest.total == 0 || beta.is_one()) return TFB_OK;
    int64_t blocks = (nest.total + 255) / 256;
    int64_t cap = (int64_t)ctx->sm_count * 16;
    int grid = (int)(blocks < cap ? blocks : cap);
    LaunchScope ls(ctx, "scale");
    launch_overlapped(ctx, scale_kernel<T>, dim3(grid), dim3(256), 0, 0u, nest, (T*)out, Ops<T>::from(beta), beta.is_zero());
    TFB_CUDA(cudaGetLastError());
    return TFB_OK;
}
tfb_status launch_scale(tfb_ctx* ctx, int dtype, const LoopNest& nest, void* out, Scalar beta) {
    DeviceGuard g(ctx->device);
    switch (dtype) {
        case TFB_F32: return scale_typed<float>(ctx, nest, out, beta);
        case TFB_F64: return scale_typed<double>(ctx, nest, out, beta);
        case TFB_C32: return scale_typed<float2>(ctx, nest, out, beta);
        case TFB_C64: return scale_typed<double2>(ctx, nest, out, beta);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

// ------------------------------------------------------------------ element-wise product
template <typename T>
__global__ void __launch_bounds__(256) ewmul_kernel(LoopNest nest, const T* a, const T* b,
                                                    T* out, EpilogueArgs<T> ep, bool conj_a, bool conj_b) {
    launch_begin();
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < nest.total; idx += stride) {
        int64_t off[3];
        decompose<3>(nest, 0, idx, off);
        T x = a[off[0]], y = b[off[1]];
        if (conj_a) x = Ops<T>::conj(x);
        if (conj_b) y = Ops<T>::conj(y);
        out[off[2]] = ep.apply(Ops<T>::mul(x, y), out + off[2]);
    }
}
// Row form: the output's mode 0 has stride 1, each input's 1 or 0.  A thread has four units (V elements, one
// access) of every tensor in flight; bound by HBM, or by latency and the launch below a few MB.  1021 x 2 x 1021
// complex double times a bond's weights: 14 us against 19 us element by element with a division per mode.
template <typename T, int V, typename N>
__global__ void __launch_bounds__(256) ewmul_rows_kernel(N nest, const T* a, const T* b, T* out, EpilogueArgs<T> ep, bool conj_a,
                                                         bool conj_b, bool run_a, bool run_b) {
    launch_begin();
    constexpr int U = 4;
    const int64_t units = nest.total / V, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t u0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u0 < units; u0 += U * stride) {
        Pack<T, V> x[U], y[U], o[U];
        T* dst[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int64_t u = u0 + k * stride;
            if (u >= units) continue;
            int64_t q, r, off[3];
            divide_inner(nest, V, u, q, r);
            decompose<3>(nest, 1, q, off);
            if (run_a) x[k] = *reinterpret_cast<const Pack<T, V>*>(a + off[0] + r * V);
            else x[k].v[0] = a[off[0]];
            if (run_b) y[k] = *reinterpret_cast<const Pack<T, V>*>(b + off[1] + r * V);
            else y[k].v[0] = b[off[1]];
            dst[k] = out + off[2] + r * V;
            if (ep.read_out) o[k] = *reinterpret_cast<const Pack<T, V>*>(dst[k]);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (u0 + k * stride >= units) continue;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                T p = x[k].v[run_a ? i : 0], w = y[k].v[run_b ? i : 0];
                if (conj_a) p = Ops<T>::conj(p);
                if (conj_b) w = Ops<T>::conj(w);
                o[k].v[i] = ep.apply(Ops<T>::mul(p, w), &o[k].v[i]);
            }
            *reinterpret_cast<Pack<T, V>*>(dst[k]) = o[k];
        }
    }
}
template <typename T, int V>
static void launch_ewmul_rows(tfb_ctx* ctx, const LoopNest& nest, const T* a, const T* b, T* out, const EpilogueArgs<T>& ep, bool ca,
                              bool cb) {
    const bool run_a = nest.stride[0][0] != 0, run_b = nest.stride[1][0] != 0;
    const unsigned grid = grid_of_four(nest.total / V, ctx->sm_count, 8);
    if (Nest32::fits(nest)) {
        Nest32 n(nest);
        n.div[0] = FastDiv::of((uint32_t)(nest.extent[0] / V));
        launch_overlapped(ctx, ewmul_rows_kernel<T, V, Nest32>, dim3(grid), dim3(256), 0, 0u, n, a, b, out, ep, ca, cb, run_a, run_b);
    } else {
        launch_overlapped(ctx, ewmul_rows_kernel<T, V, LoopNest>, dim3(grid), dim3(256), 0, 0u, nest, a, b, out, ep, ca, cb, run_a, run_b);
    }
}
// Flat form: the output and one input lie without a gap, so they move sixteen bytes at a time whatever the extents; runs of an odd
// number of elements leave the row form one element an access.  The other input is looked up: a weight per row or column,
// from L1 as a rule.  One unit a thread and turn, so that registers leave room for five blocks an SM (1999 x 4 x 2047 floats times
// a weight per row: 72 us by rows, 41 with four units a turn, 34 with two, 33 so; 1501 x 3 x 1501 doubles 34.5, 27.4).  Two
// flat inputs gain nothing (1501 x 3 x 1501 doubles 31.4 by rows, 33.5).
template <typename T, int V>
__global__ void __launch_bounds__(256, 5) ewmul_flat_kernel(Nest32 nest, const T* a, const T* b, T* out, EpilogueArgs<T> ep, bool conj_a,
                                                            bool conj_b, bool flat_a) {
    launch_begin();
    const int64_t units = nest.total / V, stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const T* whole = flat_a ? a : b;
    const T* other = flat_a ? b : a;
    const int64_t step = flat_a ? nest.stride[1][0] : nest.stride[0][0];
    auto at = [&](uint32_t i) {
        int64_t off[3];
        decompose<3>(nest, 0, i, off);
        return flat_a ? off[1] : off[0];  // (no index: the array stays in registers)
    };
    auto product = [&](T x, T w, T* old) {  // an element of `whole`, one of `other`
        T p = flat_a ? x : w, q = flat_a ? w : x;
        if (conj_a) p = Ops<T>::conj(p);
        if (conj_b) q = Ops<T>::conj(q);
        return ep.apply(Ops<T>::mul(p, q), old);
    };
    for (int64_t u = first; u < units; u += stride) {
        const Pack<T, V> x = *reinterpret_cast<const Pack<T, V>*>(whole + u * V);
        Pack<T, V> o, y;
        if (ep.read_out) o = *reinterpret_cast<const Pack<T, V>*>(out + u * V);
        const uint32_t i = (uint32_t)(u * V), q = nest.div[0].quotient(i), r = i - q * nest.div[0].d;
        int64_t off[3];
        decompose<3>(nest, 1, q, off);
        const T* src = other + (flat_a ? off[1] : off[0]) + r * step;
        if (r + V <= nest.div[0].d) {
            // neighbours in the same run are a step apart, or the same element
            if (step == 0) {
                const T one = *src;
#pragma unroll
                for (int e = 0; e < V; ++e) y.v[e] = one;
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) y.v[e] = src[e];
            }
        } else {
#pragma unroll 1
            for (int e = 0; e < V; ++e) {
                const T one = other[at(i + e)];
#pragma unroll
                for (int f = 0; f < V; ++f)
                    if (f == e) y.v[f] = one;
            }
        }
#pragma unroll
        for (int e = 0; e < V; ++e) o.v[e] = product(x.v[e], y.v[e], &o.v[e]);
        *reinterpret_cast<Pack<T, V>*>(out + u * V) = o;
    }
    const int64_t i = units * V + first;  // what is left of a unit
    if (i < nest.total) out[i] = product(whole[i], other[at((uint32_t)i)], out + i);
}
template <typename T>
static tfb_status ewmul_typed(tfb_ctx* ctx, const LoopNest& nest, const void* a, const void* b, void* out,
                              Scalar alpha, Scalar beta, bool ca, bool cb) {
    if (nest.total == 0) return TFB_OK;
    EpilogueArgs<T> ep = EpilogueArgs<T>::make(alpha, beta, false);
    int64_t blocks = (nest.total + 255) / 256;
    int64_t cap = (int64_t)ctx->sm_count * 16;
    int grid = (int)(blocks < cap ? blocks : cap);
    LaunchScope ls(ctx, "elementwise_mul");
    // Overlap between out and an input is only in order where both are walked alike, which the element
    // kernel does for any strides and the row kernel for the same ones.
    const bool rows = nest.rank >= 1 && nest.stride[2][0] == 1 && (nest.stride[0][0] == 1 || nest.stride[0][0] == 0) &&
                      (nest.stride[1][0] == 1 || nest.stride[1][0] == 0);
    if (rows) {
        constexpr int VMAX = sizeof(T) < 16 ? 16 / sizeof(T) : 1;
        // 16-byte accesses: runs of whole units, every other stride a multiple of a unit, aligned bases.
        bool vec = VMAX > 1 && nest.extent[0] % VMAX == 0;
        const void* base[3] = {a, b, out};
        for (int t = 0; t < 3 && vec; ++t) {
            if (nest.stride[t][0] == 0) continue;
            vec = (uintptr_t)base[t] % 16 == 0;
            for (int d = 1; d < nest.rank && vec; ++d) vec = nest.stride[t][d] % VMAX == 0;
        }
        // Without gaps: the strides are the extents' products.  From some 100 000 elements on; below, both are one round of latency.
        bool flat[3];
        for (int t = 0; t < 3; ++t) {
            int64_t step = 1;
            flat[t] = (uintptr_t)base[t] % 16 == 0;
            for (int d = 0; d < nest.rank && flat[t]; ++d) {
                flat[t] = nest.stride[t][d] == step;
                step *= nest.extent[d];
            }
        }
        if (!vec && VMAX > 1 && flat[2] && flat[0] != flat[1] && nest.total >= 100000 && Nest32::fits(nest)) {
            const int64_t per_pass = (nest.total / VMAX + 255) / 256;
            launch_overlapped(ctx, ewmul_flat_kernel<T, VMAX>, dim3((unsigned)std::min<int64_t>(per_pass, (int64_t)ctx->sm_count * 8)), dim3(256), 0, 0u,
                              Nest32(nest), (const T*)a, (const T*)b, (T*)out, ep, ca, cb, flat[0]);
        } else if (vec) launch_ewmul_rows<T, VMAX>(ctx, nest, (const T*)a, (const T*)b, (T*)out, ep, ca, cb);
        else launch_ewmul_rows<T, 1>(ctx, nest, (const T*)a, (const T*)b, (T*)out, ep, ca, cb);
        TFB_CUDA(cudaGetLastError());
        return TFB_OK;
    }
    launch_overlapped(ctx, ewmul_kernel<T>, dim3(grid), dim3(256), 0, 0u, nest, (const T*)a, (const T*)b, (T*)out, ep, ca, cb);
    TFB_CUDA(cudaGetLastError());
    return TFB_OK;
}
tfb_status launch_elementwise_mul(tfb_ctx* ctx, int dtype, const LoopNest& nest, const void* a, const void* b,
                                  void* out, Scalar alpha, Scalar beta, bool conj_a, bool conj_b) {
    DeviceGuard g(ctx->device);
    switch (dtype) {
        case TFB_F32: return ewmul_typed<float>(ctx, nest, a, b, out, alpha, beta, conj_a, conj_b);
        case TFB_F64: return ewmul_typed<double>(ctx, nest, a, b, out, alpha, beta, conj_a, conj_b);
        case TFB_C32: return ewmul_typed<float2>(ctx, nest, a, b, out, alpha, beta, conj_a, conj_b);
        case TFB_C64: return ewmul_typed<double2>(ctx, nest, a, b, out, alpha, beta, conj_a, conj_b);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

// ------------------------------------------------------------------ reduce
// A block is TX kept elements x G threads each, the reduced range of an element dealt out to its G
// threads in turns (times gridDim.y slices).  Neighbouring threads follow the input's unit stride:
//   RED_FAST    the G threads of an element are neighbours (unit stride in a reduced mode)
//   otherwise   neighbouring threads hold neighbouring kept elements
// Each thread has eight loads in flight whatever the inner run's length.  With several slices the partial
// results go to `partial[slice][kept]`, and the last block of a group of kept elements to arrive combines them, or
// reduce_finish_kernel where there are many.  All orders are fixed: results do not depend on scheduling.  Bound by HBM from about 20 MB on.  Before, a warp took
// one kept element (seven of eight warps idle when there was one only) and a thread of the finishing kernel
// all slices of one: 700473 x 156 f32 to a scalar 446 -> 84 us, 12 x 56 x 8810 x 17 f64 keeping the outer ones
// 307 -> 140, 27 x 38 x 11916 f64 keeping the middle 142 -> 24, 301 x 2003 x 203 keeping the outer 178 -> 158.
template <typename T, int OP>
struct Red {
    __device__ static T init() {
        if (OP == TFB_REDUCE_SUM) return Ops<T>::zero();
        if (OP == TFB_REDUCE_MAX) return Ops<T>::lowest();
        return Ops<T>::highest();
    }
    __device__ static T comb(T a, T b) {
        if (OP == TFB_REDUCE_SUM) return Ops<T>::add(a, b);
        if (OP == TFB_REDUCE_MAX) return Ops<T>::max_(a, b);
        return Ops<T>::min_(a, b);
    }
};

template <typename T>
__device__ __forceinline__ T shuffle_down(T v, int s) {
    union { T t; uint32_t w[sizeof(T) / 4]; } u;
    u.t = v;
#pragma unroll
    for (int i = 0; i < (int)sizeof(T) / 4; ++i) u.w[i] = __shfl_down_sync(0xffffffffu, u.w[i], s);
    return u.t;
}
// Combines the values of the G threads of each kept element; the result is valid where g == 0.  In the same order by
// shuffles, where the threads are neighbours in a warp, and through shared memory.
template <typename T, int OP>
__device__ __forceinline__ T combine_group(T acc, T* sh, int g, int G, int step) {
    if (G == 1) return acc;
    if (step == 1 && G <= 32) {
        for (int s = G >> 1; s > 0; s >>= 1) acc = Red<T, OP>::comb(acc, shuffle_down(acc, s));
        return acc;
    }
    __syncthreads();
    sh[threadIdx.x] = acc;
    for (int s = G >> 1; s > 0; s >>= 1) {
        __syncthreads();
        if (g < s) sh[threadIdx.x] = Red<T, OP>::comb(sh[threadIdx.x], sh[threadIdx.x + s * step]);
    }
    return sh[threadIdx.x];
}

// Walks a thread's elements r0 + g, r0 + g + G, ... of the reduced range without a division per element.
// One mode: a pointer step.  Two: a step in both with a carry.  More: the linear index by multiplication.  From 2^31
// elements on, where that would take hardware divisions: a step in the two inner modes with carries, divisions only
// when the second one wraps (f32, per launch, against a division per element and mode: 46341 x 46400 padded to a
// scalar 11.5 -> 5.2 ms, 1001 x 1500 x 1500 16.5 -> 5.4, 1300^3 x 2 keeping the last 31.9 -> 10.4).
template <int RANK, typename N>
struct RedWalk;
template <typename N>
struct RedWalk<1, N> {
    int64_t off, step;
    __device__ __forceinline__ RedWalk(const N& red, int64_t r, int G) : off(r * red.stride[0][0]), step(G * red.stride[0][0]) {}
    __device__ __forceinline__ int64_t next(const N&, int64_t, int) {
        const int64_t o = off;
        off += step;
        return o;
    }
};
template <>
struct RedWalk<2, Nest32> {
    uint32_t i0, g0, e0;
    int64_t off, step, wrap;
    __device__ __forceinline__ RedWalk(const Nest32& red, int64_t r, int G) : e0(red.div[0].d) {
        const uint32_t q = red.div[0].quotient((uint32_t)r), gq = red.div[0].quotient((uint32_t)G);
        i0 = (uint32_t)r - q * e0;
        g0 = (uint32_t)G - gq * e0;
        off = i0 * red.stride[0][0] + q * red.stride[0][1];
        step = g0 * red.stride[0][0] + gq * red.stride[0][1];
        wrap = red.stride[0][1] - (int64_t)e0 * red.stride[0][0];
    }
    __device__ __forceinline__ int64_t next(const Nest32&, int64_t, int) {
        const int64_t o = off;
        i0 += g0;
        off += step;
        if (i0 >= e0) {
            i0 -= e0;
            off += wrap;
        }
        return o;
    }
};
template <>
struct RedWalk<0, LoopNest> {
    int64_t i0, i1, q, off, outer, g0, g1, gq;
    __device__ static int64_t extent(const LoopNest& red, int d) { return d < red.rank ? red.extent[d] : 1; }
    __device__ static int64_t stride(const LoopNest& red, int d) { return d < red.rank ? red.stride[0][d] : 0; }
    __device__ __forceinline__ RedWalk(const LoopNest& red, int64_t r, int G) {
        divmod(r, extent(red, 0), q, i0);
        divmod(q, extent(red, 1), q, i1);
        divmod(G, extent(red, 0), gq, g0);
        divmod(gq, extent(red, 1), gq, g1);
        int64_t o[1];
        decompose<1>(red, 2, q, o);
        outer = o[0];
        off = i0 * stride(red, 0) + i1 * stride(red, 1) + outer;
    }
    __device__ __forceinline__ int64_t next(const LoopNest& red, int64_t, int) {
        const int64_t o = off, e0 = extent(red, 0), e1 = extent(red, 1), s0 = stride(red, 0), s1 = stride(red, 1);
        int64_t step1 = g1, step2 = gq;
        i0 += g0;
        off += g0 * s0;
        if (i0 >= e0) {
            i0 -= e0;
            off -= e0 * s0;
            ++step1;
        }
        i1 += step1;
        off += step1 * s1;
        if (i1 >= e1) {
            i1 -= e1;
            off -= e1 * s1;
            ++step2;
        }
        if (step2) {
            int64_t x[1];
            q += step2;
            decompose<1>(red, 2, q, x);
            off += x[0] - outer;
            outer = x[0];
        }
        return o;
    }
};
template <typename N>
struct RedWalk<0, N> {
    __device__ __forceinline__ RedWalk(const N&, int64_t, int) {}
    __device__ __forceinline__ int64_t next(const N& red, int64_t r, int) {
        int64_t off[1];
        decompose<1>(red, 0, r, off);
        return off[0];
    }
};

// Loads in flight per thread, and CTAs per SM that their registers leave: 48 to 64 KB per SM.
template <typename T>
constexpr int kRedLoads = sizeof(T) == 4 ? 16 : 8;
template <typename T>
constexpr int kRedCtas = sizeof(T) == 16 ? 2 : sizeof(T) == 4 ? 3 : 4;
// (the walk in 64 bits holds too many values for more than two)
template <typename T, int RANK, typename N>
constexpr int kRedBound = RANK == 0 && std::is_same<N, LoopNest>::value ? 2 : kRedCtas<T>;
// SHORT: a thread has no more than eight elements, and four loads in flight: with sixteen most of them would be
// tests and neutral elements (496 x 1576 x 16 f32, the maximum over the last index: 30 us, 14 before).
// ONE: the last block of a group combines its slices.
template <typename T, int OP, bool RED_FAST, int RANK, bool SHORT, bool ONE, typename N>
__global__ void __launch_bounds__(256, (SHORT ? 4 : kRedBound<T, RANK, N>)) reduce_kernel(const __grid_constant__ N kept, const __grid_constant__ N red,
                                                     const T* in, T* out, T* partial, unsigned* arrived, int log_g,
                                                     int64_t chunk, EpilogueArgs<T> ep) {
    launch_begin();
    constexpr int U = SHORT ? 4 : kRedLoads<T>;
    __shared__ T sh[256];
    const int G = 1 << log_g, TX = 256 >> log_g;
    const int g = RED_FAST ? threadIdx.x & (G - 1) : threadIdx.x / TX;
    const int x = RED_FAST ? threadIdx.x >> log_g : threadIdx.x & (TX - 1);
    const int64_t r0 = (int64_t)blockIdx.y * chunk, r1 = min(red.total, r0 + chunk);
    const int64_t groups = (kept.total + TX - 1) / TX;
    for (int64_t kb = blockIdx.x; kb < groups; kb += gridDim.x) {
        const int64_t ko = kb * TX + x;
        int64_t koff[2] = {0, 0};
        T part[U];
#pragma unroll
        for (int u = 0; u < U; ++u) part[u] = Red<T, OP>::init();
        if (ko < kept.total && r0 + g < r1) {
            decompose<2>(kept, 0, ko, koff);
            const T* p = in + koff[0];
            RedWalk<RANK, N> walk(red, r0 + g, G);
            int64_t r = r0 + g;
            for (; r + (U - 1) * G < r1; r += U * G) {
                T v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = p[walk.next(red, r + u * G, G)];
#pragma unroll
                for (int u = 0; u < U; ++u) part[u] = Red<T, OP>::comb(part[u], v[u]);
            }
            if (r < r1) {
                T v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = r + u * G < r1 ? p[walk.next(red, r + u * G, G)] : Red<T, OP>::init();
#pragma unroll
                for (int u = 0; u < U; ++u) part[u] = Red<T, OP>::comb(part[u], v[u]);
            }
        }
#pragma unroll
        for (int s = U / 2; s > 0; s >>= 1)
#pragma unroll
            for (int u = 0; u < s; ++u) part[u] = Red<T, OP>::comb(part[u], part[u + s]);
        const T acc = combine_group<T, OP>(part[0], sh, g, G, RED_FAST ? 1 : TX);
        if (g == 0 && ko < kept.total) {
            if (!ONE && !partial) out[koff[1]] = ep.apply(acc, out + koff[1]);
            else partial[(int64_t)blockIdx.y * kept.total + ko] = acc;
        }
        if constexpr (ONE) {
            // The block that completes a group's slices combines them, each thread its share in slice order.
            __shared__ bool last;
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                last = atomicAdd(arrived + kb, 1u) == gridDim.y - 1;
                if (last) arrived[kb] = 0;
            }
            __syncthreads();
            if (last) {
                __threadfence();
                T sum = Red<T, OP>::init();
                if (ko < kept.total) {
#pragma unroll 8
                    for (int s = g; s < (int)gridDim.y; s += G) sum = Red<T, OP>::comb(sum, __ldcg(partial + (int64_t)s * kept.total + ko));
                }
                sum = combine_group<T, OP>(sum, sh, g, G, RED_FAST ? 1 : TX);
                if (g == 0 && ko < kept.total) out[koff[1]] = ep.apply(sum, out + koff[1]);
            }
        }
    }
}

// Combines the slices of each kept element: TX elements x G threads per block, as above.
template <typename T, int OP, typename N>
__global__ void __launch_bounds__(256) reduce_finish_kernel(N kept, const T* partial, T* out, int splits, int log_g,
                                                            EpilogueArgs<T> ep) {
    launch_begin();
    __shared__ T sh[256];
    const int G = 1 << log_g, TX = 256 >> log_g, g = threadIdx.x / TX, x = threadIdx.x & (TX - 1);
    const int64_t groups = (kept.total + TX - 1) / TX;
    for (int64_t kb = blockIdx.x; kb < groups; kb += gridDim.x) {
        const int64_t ko = kb * TX + x;
        T acc = Red<T, OP>::init();
        if (ko < kept.total) {
#pragma unroll 8
            for (int s = g; s < splits; s += G) acc = Red<T, OP>::comb(acc, partial[(int64_t)s * kept.total + ko]);
        }
        acc = combine_group<T, OP>(acc, sh, g, G, TX);
        if (g == 0 && ko < kept.total) {
            int64_t koff[2];
            decompose<2>(kept, 0, ko, koff);
            out[koff[1]] = ep.apply(acc, out + koff[1]);
        }
    }
}

// How a reduction is laid out over the chip.
struct ReduceShape {
    bool red_fast;
    int log_g = 0, splits = 1;
    int64_t chunk = 0;
    unsigned grid = 1;
    bool one_launch = false;  // the last block of a group combines its slices
};
static ReduceShape reduce_shape(const tfb_ctx* ctx, const LoopNest& kept, const LoopNest& red, int ctas, int64_t max_splits) {
    // Smallest |input stride| among reduced and kept modes.
    auto min_stride = [](const LoopNest& n) {
        int64_t m = INT64_MAX;
        for (int d = 0; d < n.rank; ++d) {
            const int64_t s = n.stride[0][d] < 0 ? -n.stride[0][d] : n.stride[0][d];
            if (n.extent[d] > 1 && s < m) m = s;
        }
        return m;
    };
    ReduceShape r;
    r.red_fast = kept.rank == 0 || min_stride(red) < min_stride(kept);
    const int64_t sms = ctx->sm_count;
    int g = 1;
    if (r.red_fast) {
        // A block per element once the elements alone cannot fill the chip, a warp for long ranges, eight
        // threads (64 bytes of f64) for short ones.
        if (red.total >= 2048 && kept.total < sms * 64) g = 256;
        else g = red.total >= 64 ? 32 : 8;
    } else {
        while (g < 32 && kept.total * g <= 128) g *= 2;  // few kept elements: the rest of the block shares them
        while (g > 1 && g > red.total) g /= 2;
    }
    while ((1 << r.log_g) < g) ++r.log_g;
    // Slices only where a thread keeps 32 elements (below that the finishing launch costs more): the fewest
    // that leave no more than a fourteenth of the last wave's places empty, else the fullest.
    const int64_t tx = 256 >> r.log_g, groups = (kept.total + tx - 1) / tx, slots = sms * ctas;
    if (groups < 4 * slots) {
        const int64_t most = std::min<int64_t>(std::min<int64_t>(red.total / ((int64_t)g * 32), max_splits),
                                               std::max<int64_t>(1, 4 * slots / groups));
        double best = 0;
        for (int64_t s = 1; s <= most && best < 0.93; ++s) {
            const int64_t blocks = groups * s;
            const double full = (double)blocks / (double)((blocks + slots - 1) / slots * slots);
            if (full > best) {
                best = full;
                r.splits = (int)s;
            }
        }
    }
    r.chunk = (red.total + r.splits - 1) / r.splits;
    r.splits = (int)((red.total + r.chunk - 1) / r.chunk);
    r.grid = (unsigned)std::min<int64_t>(groups, slots * 8);
    // Up to 32 slices the last block to arrive combines them: a launch less for the host, 16.3 -> 13.4 us a call at 20 x 29 x
    // 13 x 32 f64 keeping the first two, 17.8 -> 16.5 at 119 x 62 x 465 f32 keeping the middle, and the same time on the GPU.
    // More slices, or few threads for them, keep the launch that spreads them over the chip.
    r.one_launch = r.splits > 1 && r.splits <= std::min(32, 16 * g) && groups <= (int64_t)tfb_ctx::kArrived;
    return r;
}

template <typename T, int OP, typename N>
static void reduce_launch(tfb_ctx* ctx, const N& kept, const N& red, const T* in, T* out, T* partial, const ReduceShape& r,
                          const EpilogueArgs<T>& ep) {
    const dim3 grid(r.grid, (unsigned)r.splits);
    auto go = [&](auto rank, auto few, auto one) {
        constexpr int RANK = decltype(rank)::value;
        constexpr bool SHORT = decltype(few)::value, ONE = decltype(one)::value;
        if (r.red_fast)
            launch_overlapped(ctx, reduce_kernel<T, OP, true, RANK, SHORT, ONE, N>, grid, dim3(256), 0, 0u, kept, red, in, out, partial, ctx->arrived, r.log_g, r.chunk, ep);
        else
            launch_overlapped(ctx, reduce_kernel<T, OP, false, RANK, SHORT, ONE, N>, grid, dim3(256), 0, 0u, kept, red, in, out, partial, ctx->arrived, r.log_g, r.chunk, ep);
    };
    auto by_rank = [&](auto few, auto one) {
        if (red.rank == 1) return go(std::integral_constant<int, 1>{}, few, one);
        if constexpr (std::is_same<N, Nest32>::value)
            if (red.rank == 2) return go(std::integral_constant<int, 2>{}, few, one);
        go(std::integral_constant<int, 0>{}, few, one);
    };
    // (a slice has at least 32 elements a thread: none is short)
    if (r.one_launch) return by_rank(std::false_type{}, std::true_type{});
    if constexpr (std::is_same<N, Nest32>::value)
        if (r.chunk <= (int64_t)8 << r.log_g) return by_rank(std::true_type{}, std::false_type{});
    by_rank(std::false_type{}, std::false_type{});
}
template <typename T, int OP, typename N>
static void reduce_finish_launch(tfb_ctx* ctx, const N& kept, T* out, const T* partial, const ReduceShape& r,
                                 const EpilogueArgs<T>& ep) {
    int log_g = 0;  // about eight slices per thread
    while (log_g < 8 && (r.splits >> log_g) > 8) ++log_g;
    const int64_t tx = 256 >> log_g;
    const unsigned grid = (unsigned)std::min<int64_t>((kept.total + tx - 1) / tx, (int64_t)ctx->sm_count * 32);
    launch_overlapped(ctx, reduce_finish_kernel<T, OP, N>, dim3(grid), dim3(256), 0, 0u, kept, partial, out, r.splits, log_g, ep);
}
// Both launches; `partial` holds r.splits slices when there are several.
template <typename T, int OP>
static tfb_status reduce_run(tfb_ctx* ctx, const LoopNest& kept, const LoopNest& red, const void* in, void* out, void* partial,
                             const ReduceShape& r, const EpilogueArgs<T>& ep) {
    const bool small = Nest32::fits(kept) && Nest32::fits(red);
    {
        LaunchScope ls(ctx, "reduce");
        if (small) reduce_launch<T, OP>(ctx, Nest32(kept), Nest32(red), (const T*)in, (T*)out, (T*)partial, r, ep);
        else reduce_launch<T, OP>(ctx, kept, red, (const T*)in, (T*)out, (T*)partial, r, ep);
    }
    TFB_CUDA(cudaGetLastError());
    if (r.splits > 1 && !r.one_launch) {
        LaunchScope ls(ctx, "reduce_finish");
        if (small) reduce_finish_launch<T, OP>(ctx, Nest32(kept), (T*)out, (const T*)partial, r, ep);
        else reduce_finish_launch<T, OP>(ctx, kept, (T*)out, (const T*)partial, r, ep);
    }
    TFB_CUDA(cudaGetLastError());
    return TFB_OK;
}

template <typename T, int OP>
static tfb_status reduce_typed(tfb_ctx* ctx, const LoopNest& kept, const LoopNest& red, const void* in, void* out,
                               Scalar alpha, Scalar beta, bool conj) {
    if (kept.total == 0) return TFB_OK;
    EpilogueArgs<T> ep = EpilogueArgs<T>::make(alpha, beta, conj);
    if (red.total == 0) {
        // Empty reduction: Sum gives 0; Max/Min over nothing is rejected at plan time.
        return launch_scale(ctx, std::is_same<T, float>::value    ? TFB_F32
                                 : std::is_same<T, double>::value ? TFB_F64
                                 : std::is_same<T, float2>::value ? TFB_C32
                                                                  : TFB_C64,
                            [&] {
                                LoopNest o = kept;
                                for (int d = 0; d < o.rank; ++d) o.stride[0][d] = kept.stride[1][d];
                                return o;
                            }(),
                            out, beta);
    }
    const ReduceShape r = reduce_shape(ctx, kept, red, kRedCtas<T>, INT64_MAX);
    PoolBlock ws;
    if (r.splits > 1) TFB_TRY(ws.alloc(ctx, sizeof(T) * (size_t)r.splits * (size_t)kept.total));
    return reduce_run<T, OP>(ctx, kept, red, in, out, ws.ptr, r, ep);
}

template <typename T>
static tfb_status reduce_op_dispatch(tfb_ctx* ctx, int op, const LoopNest& kept, const LoopNest& red, const void* in,
                                     void* out, Scalar alpha, Scalar beta, bool conj) {
    switch (op) {
        case TFB_REDUCE_SUM: return reduce_typed<T, TFB_REDUCE_SUM>(ctx, kept, red, in, out, alpha, beta, conj);
        case TFB_REDUCE_MAX: return reduce_typed<T, TFB_REDUCE_MAX>(ctx, kept, red, in, out, alpha, beta, conj);
        case TFB_REDUCE_MIN: return reduce_typed<T, TFB_REDUCE_MIN>(ctx, kept, red, in, out, alpha, beta, conj);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown reduce op %d", op);
}

tfb_status launch_reduce(tfb_ctx* ctx, int dtype, int op, const LoopNest& kept, const LoopNest& red, const void* in,
                         void* out, Scalar alpha, Scalar beta, bool conj) {
    DeviceGuard g(ctx->device);
    switch (dtype) {
        case TFB_F32: return reduce_op_dispatch<float>(ctx, op, kept, red, in, out, alpha, beta, conj);
        case TFB_F64: return reduce_op_dispatch<double>(ctx, op, kept, red, in, out, alpha, beta, conj);
        case TFB_C32:
            if (op != TFB_REDUCE_SUM) return fail(TFB_ERR_INVALID_ARGUMENT, "Max/Min are undefined for complex types");
            return reduce_typed<float2, TFB_REDUCE_SUM>(ctx, kept, red, in, out, alpha, beta, conj);
        case TFB_C64:
            if (op != TFB_REDUCE_SUM) return fail(TFB_ERR_INVALID_ARGUMENT, "Max/Min are undefined for complex types");
            return reduce_typed<double2, TFB_REDUCE_SUM>(ctx, kept, red, in, out, alpha, beta, conj);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", dtype);
}

// ------------------------------------------------------------------ reduce without allocation
// Some callers must not allocate device memory when they call in: an application that has
// handed all device memory to an allocator of its own, a latency-critical loop that cannot
// afford the pool's occasional trip to the driver, a framework callback in which device
// allocation is forbidden.  For them the split partials of the reduce kernel live in this
// fixed array instead of a pool block.  Every GPU that loads the library carries these
// 4 MiB until the process exits.
constexpr size_t kStaticReduceBytes = (size_t)4 << 20;
static __device__ __align__(256) unsigned char g_static_reduce_scratch[kStaticReduceBytes];

// In host code the array's name is only a handle for the runtime, not an address a kernel
// could use: the device address is asked for once per device, with that device current.
static tfb_status static_reduce_scratch(tfb_ctx* ctx, void** out) {
    static std::mutex mu;
    static std::map<int, void*> by_device;
    std::lock_guard<std::mutex> lock(mu);
    auto it = by_device.find(ctx->device);
    if (it != by_device.end()) {
        *out = it->second;
        return TFB_OK;
    }
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_reduce_scratch);
    if (e != cudaSuccess || !ptr)
        return fail(TFB_ERR_DEVICE, "cudaGetSymbolAddress(static reduce scratch) failed on device %d: %s", ctx->device,
                    cudaGetErrorString(e));
    by_device[ctx->device] = ptr;
    *out = ptr;
    return TFB_OK;
}

template <typename T, int OP>
static tfb_status reduce_static_typed(tfb_ctx* ctx, const LoopNest& kept, const LoopNest& red, const void* in, void* out,
                                      Scalar alpha, Scalar beta, bool conj, void* scratch) {
    EpilogueArgs<T> ep = EpilogueArgs<T>::make(alpha, beta, conj);
    // The partials have to fit the fixed array.
    const ReduceShape r = reduce_shape(ctx, kept, red, kRedCtas<T>, (int64_t)(kStaticReduceBytes / (sizeof(T) * (size_t)kept.total)));
    return reduce_run<T, OP>(ctx, kept, red, in, out, r.splits > 1 ? scratch : nullptr, r, ep);
}

template <typename T>
static tfb_status reduce_static_ops(tfb_ctx* ctx, int op, const LoopNest& kept, const LoopNest& red, const void* in,
                                    void* out, Scalar alpha, Scalar beta, bool conj, void* scratch) {
    switch (op) {
        case TFB_REDUCE_SUM: return reduce_static_typed<T, TFB_REDUCE_SUM>(ctx, kept, red, in, out, alpha, beta, conj, scratch);
        case TFB_REDUCE_MAX: return reduce_static_typed<T, TFB_REDUCE_MAX>(ctx, kept, red, in, out, alpha, beta, conj, scratch);
        case TFB_REDUCE_MIN: return reduce_static_typed<T, TFB_REDUCE_MIN>(ctx, kept, red, in, out, alpha, beta, conj, scratch);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown reduce op %d", op);
}

}  // namespace tfb

// See include/tenferro_b200.h.  The first call on a device looks up the scratch address
// (cudaGetSymbolAddress); after that a call is one kernel launch, two where there are more slices than one block combines, and nothing else.
extern "C" tfb_status tfb_reduce_static(tfb_ctx* ctx, int32_t dtype, int32_t reduce_op, const uint32_t* modes_a,
                                        size_t n_modes_a, const tfb_view* a, const uint32_t* modes_c, size_t n_modes_c,
                                        const tfb_view* c, const void* alpha, const void* beta) {
    using namespace tfb;
    if (!ctx || !a || !c || !alpha || !beta) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_reduce_static: NULL argument");
    if (!dtype_valid(dtype)) return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", (int)dtype);
    if (reduce_op < TFB_REDUCE_SUM || reduce_op > TFB_REDUCE_MIN)
        return fail(TFB_ERR_INVALID_ARGUMENT, "unknown reduce op %d", (int)reduce_op);
    if (reduce_op != TFB_REDUCE_SUM && dtype_is_complex(dtype))
        return fail(TFB_ERR_INVALID_ARGUMENT, "Max/Min are undefined for complex types");
    if (a->rank != n_modes_a) return fail(TFB_ERR_RANK_MISMATCH, "rank mismatch: expected %zu, got %zu (input)", n_modes_a, a->rank);
    if (c->rank != n_modes_c) return fail(TFB_ERR_RANK_MISMATCH, "rank mismatch: expected %zu, got %zu (output)", n_modes_c, c->rank);
    if ((n_modes_a && !modes_a) || (n_modes_c && !modes_c)) return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_reduce_static: modes are NULL");
    HView va, vc;
    TFB_TRY(to_hview(*a, dtype, &va, "input"));
    TFB_TRY(to_hview(*c, dtype, &vc, "output"));
    if (vc.conj) return fail(TFB_ERR_INVALID_ARGUMENT, "the output view cannot carry the conjugate flag");
    for (size_t i = 0; i < n_modes_a; ++i)
        for (size_t j = i + 1; j < n_modes_a; ++j)
            if (modes_a[i] == modes_a[j]) return fail(TFB_ERR_INVALID_ARGUMENT, "modes_a holds a repeated label");
    std::vector<Mode> kept, red;
    std::vector<bool> used(n_modes_a, false);
    for (size_t i = 0; i < n_modes_c; ++i) {
        size_t j = 0;
        while (j < n_modes_a && modes_a[j] != modes_c[i]) ++j;
        if (j == n_modes_a || used[j]) return fail(TFB_ERR_INVALID_ARGUMENT, "modes_c is not a subset of modes_a (label %u)", modes_c[i]);
        if (va.dims[j] != vc.dims[i])
            return fail(TFB_ERR_SHAPE_MISMATCH, "shape mismatch: expected [%lld], got [%lld] (label %u)", (long long)va.dims[j],
                        (long long)vc.dims[i], modes_c[i]);
        used[j] = true;
        kept.push_back(Mode{va.dims[j], {va.strides[j], vc.strides[i], 0}});
    }
    for (size_t j = 0; j < n_modes_a; ++j)
        if (!used[j]) red.push_back(Mode{va.dims[j], {va.strides[j], 0, 0}});
    int64_t kept_total = 1, red_total = 1;
    for (auto& m : kept) kept_total *= m.extent;
    for (auto& m : red) red_total *= m.extent;
    if (kept_total == 0) return TFB_OK;
    if (red_total == 0) {
        // As a Reduce plan does: the sum over nothing is 0, so C = beta * C (one launch, no
        // scratch); Max/Min over nothing have no value.
        if (reduce_op != TFB_REDUCE_SUM)
            return fail(TFB_ERR_INVALID_ARGUMENT, "tfb_reduce_static: Max/Min over an empty range is undefined");
        sort_and_fuse(kept, 1, 2);
        for (auto& m : kept) m.s[0] = m.s[1];
        LoopNest nk0;
        TFB_TRY(make_nest(kept, &nk0));
        DeviceGuard guard0(ctx->device);
        return launch_scale(ctx, dtype, nk0, vc.ptr, load_scalar(dtype, beta));
    }
    const size_t out_bytes = (size_t)kept_total * dtype_size(dtype);
    if (out_bytes > kStaticReduceBytes / 2)
        return fail(TFB_ERR_INVALID_ARGUMENT,
                    "tfb_reduce_static: the output holds %zu bytes, more than the %zu this allocation-free entry point "
                    "supports; use tfb_execute with a Reduce plan",
                    out_bytes, kStaticReduceBytes / 2);
    sort_and_fuse(kept, 1, 2);
    sort_and_fuse(red, 0, 1);
    LoopNest nk, nr;
    TFB_TRY(make_nest(kept, &nk));
    TFB_TRY(make_nest(red, &nr));
    DeviceGuard guard(ctx->device);
    void* scratch = nullptr;
    TFB_TRY(static_reduce_scratch(ctx, &scratch));
    const Scalar al = load_scalar(dtype, alpha), be = load_scalar(dtype, beta);
    switch (dtype) {
        case TFB_F32: return reduce_static_ops<float>(ctx, reduce_op, nk, nr, va.ptr, vc.ptr, al, be, va.conj, scratch);
        case TFB_F64: return reduce_static_ops<double>(ctx, reduce_op, nk, nr, va.ptr, vc.ptr, al, be, va.conj, scratch);
        case TFB_C32:
            return reduce_static_typed<float2, TFB_REDUCE_SUM>(ctx, nk, nr, va.ptr, vc.ptr, al, be, va.conj, scratch);
        case TFB_C64:
            return reduce_static_typed<double2, TFB_REDUCE_SUM>(ctx, nk, nr, va.ptr, vc.ptr, al, be, va.conj, scratch);
    }
    return fail(TFB_ERR_INVALID_ARGUMENT, "unknown dtype %d", (int)dtype);
}
