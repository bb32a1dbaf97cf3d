// C entry points to decisions that the library makes on the host, for tests/test_host_rules.py: sizes
// near 2^31 and beyond are checked here without the memory they would take.
#include "f64_map.h"

using namespace tfb;

// One operand of M x K (mn_major: rows contiguous) in a map of the given form.
// out: runs, dims[4], box[4].  Returns 1 when a map describes it.
extern "C" int f64_map(int cplx, int lines, int kr, int g, int bk, int rows, int64_t R, int64_t K, int mn_major, int64_t ld,
                       uint64_t* out) {
    ContractProblem p;
    p.dtype = cplx ? TFB_C64 : TFB_F64;
    p.k = {Mode{K, {mn_major ? ld : 1, 0, 0, 0}}};
    if (R > 1) p.m = {Mode{R, {mn_major ? 1 : ld, 0, 0, 0}}};
    F64MapShape d;
    if (!f64_map_shape(p, p.m, 0, (const void*)256, rows, F64MapForm{cplx != 0, lines != 0, kr, g, bk}, &d)) return 0;
    out[0] = d.runs;
    for (int i = 0; i < 4; ++i) {
        out[1 + i] = d.dims[i];
        out[5 + i] = d.box[i];
    }
    return 1;
}
