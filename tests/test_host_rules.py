"""Decisions of the host side at sizes no test can allocate: which operands a tensor map describes.  The rules
are plain host code (no CUDA call); tests/host_rules.cpp gives them C entry points."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "tenferro-rs_b200" / "csrc"


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = tmp_path_factory.mktemp("host_rules") / "host_rules.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-shared", "-fPIC",
                    f"-I{CSRC}", "-I/usr/local/cuda/include", str(ROOT / "tests" / "host_rules.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


# ---------------------------------------------------------------- tensor maps of the f64 / Complex64 kernel
# (complex, one load per run allowed, k per run, rows per run, k per iteration, rows per tile)
FORMS = [(1, 1, 8, 8, 32, 64), (1, 1, 8, 8, 16, 32), (1, 0, 4, 2, 32, 64), (0, 0, 4, 4, 16, 128), (0, 0, 4, 4, 16, 64)]
EDGE = 1 << 30


def f64_map(rules, form, rows, k, mn_major, ld):
    out = (C.c_uint64 * 9)()
    ok = rules.f64_map(*form, C.c_int64(rows), C.c_int64(k), int(mn_major), C.c_int64(ld), out)
    return list(out) if ok else None


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("mn_major", [False, True])
@pytest.mark.parametrize("fast", [7, 97, 4096, EDGE - 64, EDGE - 63, EDGE - 31, EDGE - 1, EDGE, EDGE + 1, EDGE + 8, 1200000001, 2**31 - 577,
                                  2**31 - 576])
def test_load_coordinates_fit_32_bits(rules, form, mn_major, fast):
    cplx, _, kr, g, bk, tile = form
    width, run, step = 1 + cplx, g if mn_major else kr, tile if mn_major else bk
    ld = fast + fast % 2  # (16-byte columns for the real forms too)
    got = f64_map(rules, form, fast if mn_major else 2, 2 if mn_major else fast, mn_major, ld)
    if got is None:
        # no map: the extent is not a number of runs, and either the form wants one or the last step's coordinate
        # would not fit
        assert fast % run and (not form[1] or (fast + step) * width > 2**31 - 1)
        return
    last = -(-fast // step) * step - run  # element at which the last load of the last step begins
    coordinate = width * last if got[0] else last // run
    assert coordinate <= 2**31 - 1
    assert bool(got[0]) == (fast % run != 0)


# ---------------------------------------------------------------- units of a grouped table
def deal(rules, dtype, table, balance):
    """[(corner of C, rows, columns, k, CTA)] of the units that a table of (m, n, k) is cut into; C's are 1 << 32 apart."""
    es, tile = {0: (4, 64), 1: (8, 64), 2: (8, 32), 3: (16, 32)}[dtype]
    words = [w for p, (m, n, k) in enumerate(table) for w in (m, n, k, 1 << 20, 1, m, 1 << 20, 1, k, (p + 1) << 32, 1, m)]
    flat = (C.c_int64 * max(1, len(words)))(*words)
    want = [(((p + 1) << 32) + (i + j * m) * es, min(tile, m - i), min(tile, n - j), k)
            for p, (m, n, k) in enumerate(table) for j in range(0, n, tile) for i in range(0, m, tile)]
    out = (C.c_int64 * (5 * (len(want) + 1)))()
    got = rules.group_units(dtype, C.c_size_t(len(table)), flat, 148, int(balance), C.c_size_t(len(want)), out)
    assert got == len(want)
    rows = [tuple(out[5 * i:5 * i + 5]) for i in range(got)]
    assert sorted(r[:4] for r in rows) == sorted(want)  # each tile once
    return rows


@pytest.mark.parametrize("dtype", [0, 1, 2, 3])
@pytest.mark.parametrize("balance", [False, True])
def test_every_tile_is_dealt_once(rules, dtype, balance):
    deal(rules, dtype, [(1 + 7 * p % 150, 1 + 11 * p % 130, 5 * p % 90) for p in range(1000)], balance)
    deal(rules, dtype, [], balance)
    deal(rules, dtype, [(0, 5, 3), (1, 1, 0), (5, 0, 3)], balance)
    # costs beyond 32 bits, among ordinary ones and alone
    for k in (2**32 - 1, 5_800_000_000, 2**34, 2**40):
        deal(rules, dtype, [(1, 1, k), (1, 1, 8), (70, 64, 64), (33, 90, k), (16, 16, 16)], balance)
        deal(rules, dtype, [(2, 3, k)], balance)


# ---------------------------------------------------------------- kernels that start while the one ahead still runs
def test_every_overlapped_kernel_waits(rules):
    """Writes of the launches ahead are visible after griddepcontrol.wait: a kernel started by launch_overlapped has it,
    unconditionally and in the body of the kernel itself.  Its inputs change while it is alive, ahead of the wait, so none
    is read as data that nobody writes (a restricted pointer to constants, __ldg)."""
    text = "\n".join(p.read_text() for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]))
    started = set(re.findall(r"launch_overlapped\(\s*ctx,\s*(\w+)", text))
    assert len(started) > 15
    bodies = {}
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        end = text.index("\n}", m.end())
        bodies[m.group(1)] = text[m.start():end]
    for kernel in started:
        assert re.search(r"^    launch_begin\(\);", bodies[kernel], re.M), kernel
        assert "__restrict__" not in bodies[kernel] and "__ldg(" not in bodies[kernel], kernel
