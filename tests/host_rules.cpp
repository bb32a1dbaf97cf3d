// C entry points to decisions that the library makes on the host, for tests/test_host_rules.py: sizes
// near 2^31 and beyond are checked here without the memory they would take.
#include "f64_map.h"
#include "grouped_layout.h"

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

// ---- units of a grouped table
namespace tfb {
tfb_status fail(tfb_status code, const char*, ...) { return code; }
}  // namespace tfb

static LayoutScratch group_scratch;

template <typename T>
static int deal(size_t n, const tfb_gemm_problem* problems, int sms, int balance, size_t cap, int64_t* out) {
    size_t bytes = 0, starts_at = 0;
    int ctas = 0;
    if (deal_units<T>(n, problems, sms, balance != 0, group_scratch, &bytes, &starts_at, &ctas) != TFB_OK) return -1;
    const GroupUnit* units = (const GroupUnit*)group_scratch.table.data();
    const int* starts = (const int*)(group_scratch.table.data() + starts_at);
    const size_t n_units = ctas ? starts_at / sizeof(GroupUnit) : 0;
    if (n_units > cap || (ctas && (starts[0] != 0 || (size_t)starts[ctas] != n_units))) return -2;
    for (int c = 0; c < ctas; ++c)
        for (int i = starts[c]; i < starts[c + 1]; ++i) {
            const int64_t row[5] = {(int64_t)units[i].c, units[i].mt, units[i].nt, units[i].k, c};
            memcpy(out + 5 * i, row, sizeof row);
        }
    return (int)n_units;
}

// out: per unit the address of its corner of C, rows, columns, k, CTA.  Returns the number of units.
extern "C" int group_units(int dtype, size_t n, const tfb_gemm_problem* problems, int sms, int balance, size_t cap, int64_t* out) {
    switch (dtype) {
        case TFB_F32: return deal<float>(n, problems, sms, balance, cap, out);
        case TFB_F64: return deal<double>(n, problems, sms, balance, cap, out);
        case TFB_C32: return deal<float2>(n, problems, sms, balance, cap, out);
    }
    return deal<double2>(n, problems, sms, balance, cap, out);
}
