"""The work this framework is measured on: what a user has it do, called as a user calls it.

Eight families of calls, over the range of sizes, element types and layouts each meets in use:

  pair      one binary contraction through a kept `ContractionTree`
  oneline   the same through `einsum_into(notation, ...)`, notation parsed and ordered per call
  chain     the left environments of an MPS transfer-matrix chain, site by site, each one kept
  network   an N-ary einsum whose intermediates stay on the device
  grouped   a table of matrix products of individual sizes (blocks of block-sparse tensors)
  permute   a tensor brought into another index order
  gauge     a site tensor scaled along a bond (element-wise product with a broadcast operand)
  reduce    a sum or maximum over some of a tensor's indices

Every tensor lies in GPU memory before the call, made from the seed; every pass writes a whole
output that the caller owns.  Tensors are column-major, the framework's default order.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tenferro-rs_b200"))

import tenferro_b200 as tb  # noqa: E402

SPACE = tb.LogicalMemorySpace.GpuMemory(0)
TORCH = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}
NUMPY = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}
SIZE = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}
# real operations of one multiply-add
FLOP = {"f32": 2, "f64": 2, "c64": 8, "c128": 8}
CHAIN = "ab,asc,bsd->cd"
NETWORK = "ijk,jlm,kmn,lnp->ip"

# Upper ends of the drawn ranges: what the largest listed case costs (f32) and what takes about
# as long at the rate of double precision (f64).
MOST_FLOPS = {"f32": 3.5e13, "f64": 4e12}
MOST_ELEMENTS = 1 << 28


def listed():
    return [
        # The smallest call: one short contraction, the one-line form, default element type.
        # Latency of the host path and of a launch or two.
        {"name": "oneline_f64_64", "family": "oneline", "dtype": "f64", "notation": "abc,bcd->ad", "dims": "64,64,64,64",
         "beta": 0.0},
        # An ordinary f32 contraction of two rank-4 tensors whose extents are no power of two and
        # no multiple of four.
        {"name": "pair_f32_ragged", "family": "pair", "dtype": "f32", "notation": "ijkl,klmn->ijmn",
         "dims": "45,43,37,31,47,41", "beta": 0.0},
        # The largest: two 4 GiB operands, 35 TFLOP.
        {"name": "pair_f32_large", "family": "pair", "dtype": "f32", "notation": "ijkl,klmn->ijmn",
         "dims": "128,128,256,256,128,128", "beta": 0.0},
        # Double precision mixed into what the output holds (the damped update of a fixed-point
        # iteration), odd extents.
        {"name": "pair_f64_mix", "family": "pair", "dtype": "f64", "notation": "ijk,kjl->il", "dims": "1531,61,33,1283",
         "beta": 0.5},
        # The environment sweep of a large MPS.
        {"name": "chain_c128_512", "family": "chain", "dtype": "c128", "chi": 512, "d": 2, "sites": 32},
        # The same at the odd bond dimensions that truncation leaves: many short dependent calls.
        {"name": "chain_c128_97", "family": "chain", "dtype": "c128", "chi": 97, "d": 2, "sites": 32},
        # A loop network in single-precision complex: large intermediates, three dependent products.
        {"name": "network_c64_96", "family": "network", "dtype": "c64", "dims": "96,96,96,96,96,96,96"},
        # A table of small products with power-of-two sizes.
        {"name": "grouped_f32_4096", "family": "grouped", "dtype": "f32", "blocks": "pow2", "problems": 4096},
        # The blocks of a block-sparse tensor pair: sizes as the symmetry sectors leave them,
        # stored back to back, double precision.
        {"name": "grouped_f64_blocks", "family": "grouped", "dtype": "f64", "blocks": "any", "problems": 1024},
        # All indices of a rank-4 tensor reversed.
        {"name": "permute_f32_reverse", "family": "permute", "dtype": "f32", "dims": "128,128,128,128", "perm": "3,2,1,0"},
        # Bond weights put back onto a site tensor.
        {"name": "gauge_c128", "family": "gauge", "dtype": "c128", "notation": "asb,b->asb", "dims": "1021,2,1021"},
        # The sum over the middle index of a rank-3 tensor.
        {"name": "reduce_f64_middle", "family": "reduce", "dtype": "f64", "dims": "301,2003,203", "kept": "0,2", "op": "Sum"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _text(values):
    return ",".join(str(v) for v in values)


def _ints(text):
    return [int(x) for x in text.split(",")]


PAIRS = ("ij,jk->ik", "ji,jk->ik", "ij,kj->ik", "ijkl,klmn->ijmn", "abc,bcd->ad", "ijk,kjl->il", "bij,bjk->bik")


def draw(rng: random.Random):
    family = rng.choice(("pair", "pair", "pair", "oneline", "chain", "network", "grouped", "grouped", "permute", "permute",
                         "gauge", "reduce"))
    if family in ("pair", "oneline"):
        dtype = rng.choice(("f32", "f64"))
        notation = rng.choice(PAIRS)
        # one size sets the work (over the whole range for kept trees, the small calls for the
        # one-line form); the extents of the labels scatter around it
        labels = _labels(notation)
        most = MOST_FLOPS[dtype] if family == "pair" else 1e9
        while True:
            flops = math.exp(rng.uniform(math.log(1e5), math.log(most)))
            side = (flops / 2) ** (1 / len(labels))
            dims = [max(2, int(side * math.exp(rng.uniform(-0.7, 0.7)))) for _ in labels]
            if rng.random() < 0.4:  # 4-element granules, as often as not
                dims = [-(-x // 4) * 4 for x in dims]
            case = {"family": family, "dtype": dtype, "notation": notation, "dims": _text(dims),
                    "beta": rng.choice((0.0, 0.0, 0.5))}
            elements = [math.prod(s) for s in _shapes(notation, dims)]
            if work(case)["flops"] <= most and max(elements) <= 1 << 30:
                return case
    if family == "chain":
        chi = _log(rng, 16, 512)
        return {"family": family, "dtype": rng.choice(("f64", "c128")), "chi": chi, "d": rng.choice((2, 2, 3, 4)),
                "sites": rng.randrange(8, 33)}
    if family == "network":
        side = _log(rng, 16, 88)
        return {"family": family, "dtype": "c64", "dims": _text(max(8, min(96, int(side * rng.uniform(0.8, 1.25)))) for _ in range(7))}
    if family == "grouped":
        return {"family": family, "dtype": rng.choice(("f32", "f64")), "blocks": rng.choice(("pow2", "any")),
                "problems": _log(rng, 64, 4096)}
    if family == "permute":
        rank = rng.randrange(2, 7)
        dims = _spread(rng, rank, _log(rng, 1 << 14, MOST_ELEMENTS // 2))
        perm = list(range(rank))
        while perm == sorted(perm):
            rng.shuffle(perm)
        return {"family": family, "dtype": rng.choice(("f32", "f64", "c128")), "dims": _text(dims), "perm": _text(perm)}
    if family == "gauge":
        chi, chi2 = _log(rng, 32, 2048), _log(rng, 32, 2048)
        return {"family": family, "dtype": rng.choice(("f32", "f64", "c128")),
                "notation": rng.choice(("asb,b->asb", "a,asb->asb", "asb,asb->asb")),
                "dims": _text((chi, rng.choice((2, 3, 4)), chi2))}
    rank = rng.randrange(2, 5)
    dims = _spread(rng, rank, _log(rng, 1 << 14, MOST_ELEMENTS // 2))
    kept = sorted(rng.sample(range(rank), rng.randrange(0, rank)))
    return {"family": "reduce", "dtype": rng.choice(("f32", "f64")), "dims": _text(dims), "kept": _text(kept) if kept else "",
            "op": rng.choice(("Sum", "Sum", "Max"))}


def _spread(rng, rank, total):
    """`rank` extents, odd ones among them, with a product of about `total`."""
    cuts = [rng.uniform(0.4, 1.6) for _ in range(rank)]
    scale = math.log(total) / sum(cuts)
    dims = [max(2, int(math.exp(c * scale))) for c in cuts]
    return dims if math.prod(dims) <= MOST_ELEMENTS else [max(2, x // 2) for x in dims]


def _labels(notation):
    return sorted(set(notation) - set(",->"))


def _shapes(notation, dims):
    extent = dict(zip(_labels(notation), dims))
    ins, out = notation.split("->")
    return [[extent[c] for c in t] for t in ins.split(",") + [out]]


def _block_sizes(case, seed):
    rng = np.random.default_rng(seed)
    if case["blocks"] == "pow2":
        return rng.choice(np.array([16, 32, 64, 128]), size=(case["problems"], 3))
    # sector dimensions: many small ones, few large ones
    return np.exp(rng.uniform(np.log(4.0), np.log(160.0), size=(case["problems"], 3))).astype(int)


def _chain_pairs(case):
    chi, d = case["chi"], case["d"]
    return 2.0 * chi * chi * d * chi  # multiply-adds of the two products of a site


def _cheapest(terms, out, extent):
    """Multiply-adds of the cheapest order of pairwise contractions."""
    if len(terms) == 1:
        return 0
    best = math.inf
    for i in range(len(terms)):
        for j in range(i):
            rest = [t for n, t in enumerate(terms) if n not in (i, j)]
            both = terms[i] | terms[j]
            keep = both & (out.union(*rest))
            best = min(best, math.prod(extent[c] for c in both) + _cheapest(rest + [keep], out, extent))
    return best


def work(case):
    family, dtype = case["family"], case["dtype"]
    es = SIZE[dtype]
    if family in ("pair", "oneline", "gauge"):
        dims = _ints(case["dims"])
        shapes = _shapes(case["notation"], dims)
        n = sum(math.prod(s) for s in shapes) + (math.prod(shapes[-1]) if case.get("beta") else 0)
        ops = FLOP[dtype] * math.prod(dims) if family != "gauge" else FLOP[dtype] / 2 * math.prod(dims)
        return {"bytes": es * n, "flops": ops}
    if family == "chain":
        chi, d, sites = case["chi"], case["d"], case["sites"]
        return {"bytes": es * (sites * chi * d * chi + (sites + 1) * chi * chi), "flops": FLOP[dtype] * sites * _chain_pairs(case)}
    if family == "network":
        dims = _ints(case["dims"])
        extent = dict(zip(_labels(NETWORK), dims))
        size = sum(math.prod(x) for x in _shapes(NETWORK, dims))
        ins, out = NETWORK.split("->")
        return {"bytes": es * size, "flops": FLOP[dtype] * _cheapest([set(t) for t in ins.split(",")], set(out), extent)}
    if family == "grouped":
        t = _block_sizes(case, 0).astype(np.float64)
        m, n, k = t[:, 0], t[:, 1], t[:, 2]
        return {"bytes": float(es * (m * k + k * n + m * n).sum()), "flops": float(2 * (m * n * k).sum())}
    dims = _ints(case["dims"])
    total = math.prod(dims)
    if family == "permute":
        return {"bytes": 2 * es * total, "flops": 0}
    kept = math.prod([dims[i] for i in _ints(case["kept"])] if case["kept"] else [1])
    return {"bytes": es * (total + kept), "flops": total}


def tolerance(case):
    family, dtype = case["family"], case["dtype"]
    if family == "permute" or (family == "reduce" and case["op"] == "Max"):
        return "exact"
    if family == "gauge":
        return {"rel": 2e-7 if dtype == "f32" else 4e-16}
    # Four times the distance from the same path in 64 bits (f32, c64: 1.7e-6, the network's three
    # dependent products 3.7e-6, reductions 2e-7) or, for double precision, from its sums in another
    # order (contractions 2e-15, chains 4e-15, reductions 4e-16).
    if dtype in ("f32", "c64"):
        return {"rel": 1.5e-5 if family == "network" else 1e-6 if family == "reduce" else 1e-5}
    return {"rel": 2e-15 if family == "reduce" else 1.5e-14}


def _random(shape, dtype, gen, scale=1.0):
    """Column-major N(0, scale^2) tensor (real and imaginary parts alike): (framework view, torch storage)."""
    n = math.prod(shape)
    real = {"c64": torch.float32, "c128": torch.float64}.get(dtype)
    if real is None:
        flat = torch.randn(n, device="cuda", dtype=TORCH[dtype], generator=gen)
    else:
        flat = torch.view_as_complex(torch.randn(n, 2, device="cuda", dtype=real, generator=gen))
    if scale != 1.0:
        flat *= scale
    return _wrap(flat, shape, dtype)


def _wrap(flat, shape, dtype):
    view = tb.Tensor.from_device_pointer(flat.data_ptr(), flat.numel() * SIZE[dtype], shape, NUMPY[dtype], SPACE, flat)
    return view, flat


def _output(shape, dtype):
    return _wrap(torch.zeros(math.prod(shape), device="cuda", dtype=TORCH[dtype]), shape, dtype)


def prepare(case, seed):
    family, dtype = case["family"], case["dtype"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    s = {"family": family, "case": case}
    if family in ("pair", "oneline", "gauge"):
        shapes = _shapes(case["notation"], _ints(case["dims"]))
        s["operands"] = [_random(x, dtype, gen)[0] for x in shapes[:-1]]
        s["beta"] = case.get("beta", 0.0)
        # a mixed output starts from values of its own
        s["out"], s["flat"] = _random(shapes[-1], dtype, gen) if s["beta"] else _output(shapes[-1], dtype)
        if family != "oneline":
            s["tree"] = tb.ContractionTree.optimize(tb.Subscripts.parse(case["notation"]), shapes[:-1])
    elif family == "chain":
        chi, d = case["chi"], case["d"]
        shape = (chi, d, chi)
        # N(0, 1/(2 chi)) or N(0, 1/chi) entries keep the environment's norm near d^sites
        scale = (1.0 / ((2.0 if dtype == "c128" else 1.0) * chi)) ** 0.5
        s["sites"] = []
        for _ in range(case["sites"]):
            site = _random(shape, dtype, gen, scale)[0]
            s["sites"].append((site, site.into_conj()))
        s["env"] = _random((chi, chi), dtype, gen)[0]
        s["envs"] = [_output((chi, chi), dtype) for _ in s["sites"]]
        s["tree"] = tb.ContractionTree.optimize(tb.Subscripts.parse(CHAIN), [(chi, chi), shape, shape])
    elif family == "network":
        shapes = _shapes(NETWORK, _ints(case["dims"]))
        s["operands"] = [_random(x, dtype, gen)[0] for x in shapes[:-1]]
        s["beta"] = 0.0
        s["out"], s["flat"] = _output(shapes[-1], dtype)
        s["tree"] = tb.ContractionTree.optimize(tb.Subscripts.parse(NETWORK), shapes[:-1])
    elif family == "grouped":
        # the table belongs to the tensors' structure, the same for every seed; the entries are the seed's
        table = _block_sizes(case, 0)
        m, n, k = table[:, 0], table[:, 1], table[:, 2]
        es = SIZE[dtype]
        offs = [np.concatenate(([0], np.cumsum(x * y))) for x, y in ((m, k), (k, n), (m, n))]
        a, b = (torch.rand(int(o[-1]), device="cuda", dtype=TORCH[dtype], generator=gen) * 2 - 1 for o in offs[:2])
        s["flat"] = torch.zeros(int(offs[2][-1]), device="cuda", dtype=TORCH[dtype])
        s["keep"] = (a, b)
        pa, pb, pc = a.data_ptr(), b.data_ptr(), s["flat"].data_ptr()
        rows = zip(m.tolist(), n.tolist(), k.tolist(), offs[0].tolist(), offs[1].tolist(), offs[2].tolist())
        problems = [(i, j, l, pa + oa * es, 1, i, pb + ob * es, 1, l, pc + oc * es, 1, i) for i, j, l, oa, ob, oc in rows]
        s["plan"] = tb.PreparedGroupedGemm(problems, NUMPY[dtype])
    else:
        dims = _ints(case["dims"])
        modes = list(range(len(dims)))
        view, flat = _random(dims, dtype, gen)
        if family == "reduce":
            flat.abs_()  # weights: their sum does not cancel
        s["operands"] = [view]
        if family == "permute":
            perm = _ints(case["perm"])
            shape = [dims[i] for i in perm]
            desc = tb.PrimDescriptor.Permute(modes, perm)
        else:
            kept = _ints(case["kept"]) if case["kept"] else []
            shape = [dims[i] for i in kept]
            desc = tb.PrimDescriptor.Reduce(modes, kept, tb.ReduceOp[case["op"]])
        s["out"], s["flat"] = _output(shape, dtype)
        s["plan"] = tb.CudaBackend.plan(desc, [dims, shape], NUMPY[dtype])
    torch.cuda.synchronize()  # the framework enqueues on its context's stream, torch on its own
    return s


def run(s):
    family, case = s["family"], s["case"]
    if family == "chain":
        env = s["env"]
        for (site, conj), (out, _) in zip(s["sites"], s["envs"]):
            tb.einsum_with_plan_into(s["tree"], [env, site, conj], 1.0, 0.0, out)
            env = out
        return [flat for _, flat in s["envs"]]
    if family == "grouped":
        s["plan"].run()
    elif family in ("permute", "reduce"):
        tb.CudaBackend.execute(s["plan"], 1.0, s["operands"], 0.0, s["out"])
    else:
        if family == "oneline":
            tb.einsum_into(case["notation"], s["operands"], 1.0, s["beta"], s["out"])
        else:
            tb.einsum_with_plan_into(s["tree"], s["operands"], 1.0, s["beta"], s["out"])
    return s["flat"]
