// How the general grouped kernel's table of problems is cut into units and dealt to CTAs: host code
// without a CUDA call (grouped.cu uploads what it makes).
#pragma once
#include <algorithm>
#include <vector>

#include "common.h"

namespace tfb {

constexpr int kGroupK = 32;     // depth of a stage
constexpr int kGroupRecs = 16;  // unit records a CTA holds in shared memory

// One output tile of one problem: pointers already moved to the tile's corner.
struct __align__(16) GroupUnit {
    const char* a;
    const char* b;
    char* c;
    int64_t a_rs, a_cs, b_rs, b_cs, c_rs, c_cs;  // elements
    int64_t k;
    uint16_t mt, nt;
    // bits 0-1: log2(warp rows); 2-3: 16-row blocks per warp; 4-7: 8-column blocks per warp (the
    // tensor-pipe forms); kAFast / kBFast: the shared tile is k-fast; kAVec / kBVec: 16-byte chunks
    uint32_t shape;
};
constexpr uint32_t kAFast = 1u << 8, kBFast = 1u << 9, kAVec = 1u << 10, kBVec = 1u << 11;
constexpr int kGroupRecChunks = (int)sizeof(GroupUnit) / 16;
static_assert(sizeof(GroupUnit) % 16 == 0, "records travel as 16-byte chunks");

// Shared tiles are [row][PK] (k fast) or [k][PM] (row fast), following the operand's unit stride.  The
// pitches keep a fragment read (half a warp of 8-byte, a quarter of 16-byte accesses) on distinct
// banks.  CTAS x STAGES x tile fill an SM's shared memory.
template <typename T>
struct GroupCfg;
template <> struct GroupCfg<double>  { static constexpr int TILE = 64, PK = 36, PM = 68, STAGES = 2, CTAS = 3, NI = 2, NJ = 4; };
template <> struct GroupCfg<double2> { static constexpr int TILE = 32, PK = 36, PM = 34, STAGES = 2, CTAS = 3, NI = 2, NJ = 2; };
template <> struct GroupCfg<float>   { static constexpr int TILE = 64, PK = 36, PM = 68, STAGES = 3, CTAS = 4, NI = 4, NJ = 8; };
template <> struct GroupCfg<float2>  { static constexpr int TILE = 32, PK = 36, PM = 36, STAGES = 3, CTAS = 4, NI = 2, NJ = 4; };

// Host buffers of the layout below, kept per thread: a one-shot call would spend as long faulting fresh
// pages in as on the layout itself.  Given back above kKeep bytes.
struct LayoutScratch {
    struct Key { uint32_t cost, problem, m_tile, n_tile; uint16_t mt, nt; uint32_t split; };
    static constexpr size_t kKeep = (size_t)4 << 20;
    std::vector<Key> keys;
    std::vector<uint32_t> order, owner;
    std::vector<char> table;
    void trim() {
        if (table.capacity() > kKeep) std::vector<char>().swap(table);
        if (keys.capacity() * sizeof(Key) > kKeep) {
            std::vector<Key>().swap(keys);
            std::vector<uint32_t>().swap(order);
            std::vector<uint32_t>().swap(owner);
        }
    }
};

// How the four warps tile a unit of mt x nt: the split with the fewest MMAs for the slowest warp.
template <typename Cfg>
uint32_t warp_split(int mt, int nt, int* mmas) {
    const int rows16 = (mt + 15) / 16, cols8 = (nt + 7) / 8;
    int lw = 1, ni = (rows16 + 1) / 2, nj = (cols8 + 1) / 2;
    for (int w = 0; w <= 2; w += 2) {  // 1 x 4 and 4 x 1 warps
        const int i = (rows16 + (1 << w) - 1) >> w, j = (cols8 + (4 >> w) - 1) >> (2 - w);
        if (i <= Cfg::NI && j <= Cfg::NJ && i * j < ni * nj) { lw = w; ni = i; nj = j; }
    }
    *mmas = ni * nj;
    return (uint32_t)(lw | (ni << 2) | (nj << 4));
}

// `balance`: a plan that will run again is worth a closer balance (1024 f64 blocks: 29 us a run against 34
// with the units dealt back and forth) and twice the time on the host.
template <typename T>
tfb_status deal_units(size_t n, const tfb_gemm_problem* problems, int sm_count, bool balance, LayoutScratch& scratch, size_t* table_bytes,
                      size_t* starts_at, int* n_ctas) {
    using Cfg = GroupCfg<T>;
    constexpr int64_t TILE = Cfg::TILE, ES = sizeof(T), V = 16 / ES;
    auto& keys = scratch.keys;
    keys.clear();
    // Costs, in units of half an m16n8k8 of the slowest warp: the arithmetic, a stage's requests and
    // barrier, and what a unit costs whatever its size.  Bucketed with an eighth's resolution.
    auto bucket = [](uint64_t c) -> uint32_t {
        if (c < 8) return (uint32_t)c;
        const int e = 63 - __builtin_clzll(c);
        return std::min<uint32_t>(255, (uint32_t)(e - 2) * 8 + (uint32_t)(c >> (e - 3) & 7));
    };
    uint32_t count[256] = {0};
    for (size_t p = 0; p < n; ++p) {
        const auto& q = problems[p];
        if (q.m <= 0 || q.n <= 0) continue;
        const int64_t tm = (q.m + TILE - 1) / TILE, tn = (q.n + TILE - 1) / TILE, steps = (q.k + 7) / 8;
        const int64_t stages = std::max<int64_t>(1, (q.k + kGroupK - 1) / kGroupK);
        if (keys.size() + (size_t)tm * (size_t)tn >= (size_t)INT32_MAX || p > UINT32_MAX)
            return fail(TFB_ERR_INVALID_ARGUMENT, "the table has too many output tiles");
        for (int64_t tj = 0; tj < tn; ++tj)
            for (int64_t ti = 0; ti < tm; ++ti) {
                const int mt = (int)std::min(TILE, q.m - ti * TILE), nt = (int)std::min(TILE, q.n - tj * TILE);
                int mmas;
                const uint32_t split = warp_split<Cfg>(mt, nt, &mmas);
                // (clamped here: counting and placing below have to see the same value)
                const uint64_t cost = std::min<uint64_t>((uint64_t)(steps * mmas * 2 + stages * (8 + (mt + nt) / 8) + 16 + mmas * 2), UINT32_MAX);
                ++count[bucket(cost)];
                keys.push_back({(uint32_t)cost, (uint32_t)p, (uint32_t)ti, (uint32_t)tj, (uint16_t)mt,
                                (uint16_t)nt, split});
            }
    }
    *n_ctas = 0;
    const size_t n_units = keys.size();
    if (n_units == 0) return TFB_OK;
    // longest first
    uint32_t at[256], sum = 0;
    for (int c = 255; c >= 0; --c) { at[c] = sum; sum += count[c]; }
    auto& order = scratch.order;
    auto& owner = scratch.owner;
    order.resize(n_units);
    owner.resize(n_units);
    for (size_t i = 0; i < n_units; ++i) order[at[bucket(keys[i].cost)]++] = (uint32_t)i;
    const size_t grid = std::min<size_t>(n_units, (size_t)sm_count * Cfg::CTAS);
    std::vector<int> starts(grid + 1, 0);
    if (balance) {
        // each to the CTA with the least work so far: the top of a heap of work << 16 | CTA
        std::vector<uint64_t> heap(grid);
        for (size_t c = 0; c < grid; ++c) heap[c] = c;
        for (size_t i = 0; i < n_units; ++i) {
            owner[i] = (uint32_t)(heap[0] & 0xffff);
            const uint64_t top = heap[0] + ((uint64_t)keys[order[i]].cost << 16);
            size_t h = 0;
            for (size_t child; (child = 2 * h + 1) < grid; h = child) {
                child += child + 1 < grid && heap[child + 1] < heap[child];
                if (heap[child] >= top) break;
                heap[h] = heap[child];
            }
            heap[h] = top;
        }
    } else {
        for (size_t i = 0, c = 0, band = 0; i < n_units; ++i) {
            owner[i] = (uint32_t)(band & 1 ? grid - 1 - c : c);
            if (++c == grid) { c = 0; ++band; }
        }
    }
    for (size_t i = 0; i < n_units; ++i) ++starts[owner[i] + 1];
    for (size_t c = 0; c < grid; ++c) starts[c + 1] += starts[c];
    const size_t unit_bytes = n_units * sizeof(GroupUnit), bytes = unit_bytes + starts.size() * sizeof(int);
    if (scratch.table.size() < bytes) scratch.table.resize(bytes);
    char* table = scratch.table.data();
    memcpy(table + unit_bytes, starts.data(), starts.size() * sizeof(int));
    GroupUnit* dealt = reinterpret_cast<GroupUnit*>(table);
    for (size_t i = 0; i < n_units; ++i) {
        const auto& key = keys[order[i]];
        const auto& q = problems[key.problem];
        const int64_t m0 = key.m_tile * TILE, n0 = key.n_tile * TILE;
        GroupUnit& u = dealt[starts[owner[i]]++];
        u.a = (const char*)q.a + m0 * q.a_rs * ES;
        u.b = (const char*)q.b + n0 * q.b_cs * ES;
        u.c = (char*)q.c + (m0 * q.c_rs + n0 * q.c_cs) * ES;
        u.a_rs = q.a_rs; u.a_cs = q.a_cs; u.b_rs = q.b_rs; u.b_cs = q.b_cs; u.c_rs = q.c_rs; u.c_cs = q.c_cs;
        u.k = q.k;
        u.mt = key.mt;
        u.nt = key.nt;
        auto vec = [&](const void* base, int64_t unit, int64_t other) {
            return V > 1 && unit == 1 && other % V == 0 && (uintptr_t)base % 16 == 0;
        };
        u.shape = key.split;
        // the shared tile follows whichever direction of the operand has the smaller stride
        if (std::llabs(q.a_cs) < std::llabs(q.a_rs)) u.shape |= kAFast | (vec(q.a, q.a_cs, q.a_rs) ? kAVec : 0);
        else u.shape |= vec(q.a, q.a_rs, q.a_cs) ? kAVec : 0;
        if (std::llabs(q.b_rs) < std::llabs(q.b_cs)) u.shape |= kBFast | (vec(q.b, q.b_rs, q.b_cs) ? kBVec : 0);
        else u.shape |= vec(q.b, q.b_cs, q.b_rs) ? kBVec : 0;
    }
    *table_bytes = bytes;
    *starts_at = unit_bytes;
    *n_ctas = (int)grid;
    return TFB_OK;
}

}  // namespace tfb
