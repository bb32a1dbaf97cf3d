// Shape of the tensor map of one operand of the TMA-fed f64 / Complex64 kernel: host arithmetic
// without a CUDA call, so that the limits of a map can be checked without a device.
#pragma once
#include "common.h"

namespace tfb {

// What a kernel configuration asks for: runs of `kr` k (K-major) or `g` rows (MN-major), `bk` k per iteration;
// `lines`: an extent that no run divides may be walked with one load per run.
struct F64MapForm {
    bool cplx, lines;
    int kr, g, bk;
};
struct F64MapShape {
    bool mn_major, runs;  // runs: one load per run, dimension 0 is the whole extent
    uint64_t dims[4], strides[3];
    uint32_t box[4];
};

// Operand `tns` of `p` with free group `fr`, tiles of `rows` rows; false when no map describes it.
inline bool f64_map_shape(const ContractProblem& p, const std::vector<Mode>& fr, int tns, const void* base, int rows,
                          const F64MapForm& f, F64MapShape* out) {
    if (fr.size() > 1 || p.k.size() != 1 || p.batch.size() > 1) return false;
    const int W = f.cplx ? 2 : 1;  // doubles per element
    const int64_t R = fr.empty() ? 1 : fr[0].extent, rs = fr.empty() ? 0 : fr[0].s[tns];
    const int64_t K = p.k[0].extent, ks = p.k[0].s[tns];
    const int64_t B = p.batch.empty() ? 1 : p.batch[0].extent, bs = p.batch.empty() ? 0 : p.batch[0].s[tns];
    if ((uintptr_t)base % 16 != 0) return false;
    auto ok16 = [&](int64_t s) { return s > 0 && (s * W * 8) % 16 == 0; };
    if (B > 1 && !ok16(bs)) return false;
    // The unit-stride index (extent `fast`, runs of `run` elements, `step` of them per k-iteration) and the other one.
    int64_t fast, slow, slow_stride;
    int run, step, slow_box;
    if (ks == 1 && (f.lines || K % f.kr == 0) && (R == 1 || ok16(rs))) {
        out->mn_major = false;
        fast = K; run = f.kr; step = f.bk;
        slow = R; slow_stride = R == 1 ? K : rs; slow_box = rows;
    } else if (rs == 1 && (f.lines || R % f.g == 0) && R > 1 && (K == 1 || ok16(ks))) {
        out->mn_major = true;
        fast = R; run = f.g; step = rows;
        slow = K; slow_stride = K == 1 ? R : ks; slow_box = f.bk;
    } else {
        return false;
    }
    out->runs = fast % run != 0;
    // Dimension 0 counts doubles, and a load's coordinate along it is a 32-bit integer: up to a whole step past the
    // last element.  (Where runs divide the extent it counts runs, in dimension 2.)
    if (out->runs && (fast + step) * W > INT32_MAX) return false;
    out->dims[0] = (uint64_t)((out->runs ? fast : run) * W);
    out->dims[1] = (uint64_t)slow;
    out->dims[2] = (uint64_t)(out->runs ? 1 : fast / run);
    out->dims[3] = (uint64_t)B;
    out->strides[0] = (uint64_t)(slow_stride * W * 8);
    out->strides[1] = (uint64_t)(run * W * 8);
    out->strides[2] = (uint64_t)(B > 1 ? bs * W * 8 : 16);
    out->box[0] = (uint32_t)(run * W);
    out->box[1] = (uint32_t)slow_box;
    out->box[2] = (uint32_t)(out->runs ? 1 : step / run);
    out->box[3] = 1;
    for (int i = 0; i < 3; ++i)
        if (out->strides[i] % 16 != 0 || out->strides[i] >= (1ull << 40)) return false;
    for (int i = 0; i < 4; ++i)
        if (out->dims[i] == 0 || out->dims[i] > 0xffffffffull) return false;
    return true;
}

}  // namespace tfb
