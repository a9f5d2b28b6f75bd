"""Measured cases: what a program on one GPU asks of this framework.

Every case goes through the classes that programs use: a plan built from a matrix, an operator built from the plan,
and the operator run again and again (`SddmmSpmmStep`, `DistSDDMM`, `DistSpMM`, `GatLayer`, and the fused kernels of
a whole mesh in lock step on one GPU, as `cli/emulate.py` runs them).  A case is

    op      "sddmm"  C = S o (A B^T)
            "spmm"   Y = beta Y + S X
            "step"   the SDDMM and then the SpMM of one matrix (the unit of bench.py)
            "gat"    Y = (S o (A B^T)) X, the attention-style chain
            "mesh"   the fused SDDMM and SpMM kernels of every rank of `mesh`
            "e2e"    a step whose dense operands start in pinned host memory
    matrix  a generator string (`utils.generate.from_spec`)
    k       width of the dense operands, over all Z layers of a mesh
    f64     values of 64 bits instead of 32
    beta    (spmm) factor of the previous result

The matrix families and the widths are those of bench.py, of cli.sweep and of the tests.  The pattern of the sparse
matrix belongs to the case; its values, the dense operands and the previous result are functions of the seed.
"""
import math

import numpy as np
import torch

from spcomm3d_b200.models.dist_ops import DistSDDMM, DistSpMM
from spcomm3d_b200.models.layer import GatLayer, SddmmSpmmStep
from spcomm3d_b200.ops.fused import FusedSDDMM, FusedSpMM, run_lockstep
from spcomm3d_b200.parallel.mesh import Mesh3D, split_k
from spcomm3d_b200.parallel.plan import build_all_plans, build_my_plan
from spcomm3d_b200.parallel.symm import LocalFabric
from spcomm3d_b200.utils import generate


def _case(op, matrix, k, f64=False, **more):
    return {"op": op, "matrix": matrix, "k": k, "f64": f64, **more}


def listed():
    return [
        # the plumbing configuration of the tests: two calls of a few microseconds, bound by launches and host work
        {"name": "step uniform-4k k32 f64", **_case("step", "uniform:4096:4096:16", 32, True)},
        # one attention head on a sampled neighbourhood, the batch size of mini-batch training
        {"name": "gat zipf-16k k64", **_case("gat", "zipf:16384:131072:1.8:4096", 64)},
        # a width that is no multiple of a 16-byte vector
        {"name": "sddmm rmat-14 k50", **_case("sddmm", "rmat:14:16", 50)},
        # an odd width, a graph with hub rows, the result added to what is there
        {"name": "spmm rmat-17 k33 beta", **_case("spmm", "rmat:17:16", 33, beta=0.5)},
        # the sweep's narrowest width on a power-law graph whose operands nearly fit the L2 cache
        {"name": "step rmat-20 k32", **_case("step", "rmat:20:16", 32)},
        # 64-bit values, a ragged number of rows, accumulation over the iterations of a solver
        {"name": "spmm er-300k k64 f64", **_case("spmm", "er:300007:300007:24", 64, True, beta=1.0)},
        # graph without structure or reuse, both kernels
        {"name": "sddmm er-1M k64", **_case("sddmm", "er:1048576:1048576:32", 64)},
        {"name": "spmm er-1M k128", **_case("spmm", "er:1048576:1048576:32", 128, beta=0.0)},
        # the rectangular power-law attention layer, an eighth of the size that the sweeps use, at their full width
        {"name": "gat zipf-256k k256", **_case("gat", "zipf:262144:2097152:1.8:4096", 256)},
        # the headline: bench.py's default workload
        {"name": "step rmat-22 k128", **_case("step", "rmat:22:16", 128)},
        # the kernels of a multi-GPU run, all eight ranks of the default mesh on one GPU
        {"name": "mesh 2x2x2 rmat-16 k128", **_case("mesh", "rmat:16:16", 128, mesh="2x2x2")},
        # operands that arrive from the host at every step
        {"name": "e2e rmat-16 k64", **_case("e2e", "rmat:16:16", 64)},
    ]


_NNZ_MIN, _NNZ_MAX = 1 << 12, 1 << 24      # nonzeros of a drawn matrix
_GATHER_MAX = 9e9                          # nonzeros x row bytes of a drawn case
_DENSE_MAX = 2.5e9                         # bytes of one dense operand of a drawn case
_MESH_NNZ_MAX = 1 << 21


def draw(rng):
    op = rng.choices(("sddmm", "spmm", "step", "gat", "mesh", "e2e"), (26, 26, 20, 16, 8, 4))[0]
    f64 = rng.random() < 0.2
    es = 8 if f64 else 4
    # half of the widths are the usual ones, the others anything in between
    k = rng.choice((16, 32, 48, 64, 96, 128, 192, 256)) if rng.random() < 0.5 else int(round(math.exp(rng.uniform(math.log(4), math.log(256)))))
    top = min(_MESH_NNZ_MAX if op in ("mesh", "e2e") else _NNZ_MAX, _GATHER_MAX / (k * es))
    nnz = math.exp(rng.uniform(math.log(_NNZ_MIN), math.log(top)))
    kind = rng.choice(("rmat", "zipf", "er", "uniform"))
    if kind == "rmat":
        ef = rng.choice((8, 16, 16, 24))
        matrix = "rmat:%d:%d" % (max(8, round(math.log2(nnz / ef))), ef)
    elif kind == "zipf":
        rows = max(64, int(nnz / 22))
        cols = int(min(rows * rng.uniform(1, 8), _DENSE_MAX / (k * es)))
        matrix = "zipf:%d:%d:1.8:%d" % (rows, cols, min(4096, cols // 2))
    else:
        degree = rng.randint(4, 40)
        rows = max(64, int(nnz / degree))
        cols = max(64, int(rows * rng.choice((1.0, 1.0, 0.5, 2.0))))
        matrix = "%s:%d:%d:%d" % (kind, rows, cols, degree)
    more = {}
    if op == "spmm":
        more["beta"] = rng.choice((0.0, 0.0, 0.0, 0.5, 1.0))
    if op == "mesh":
        more["mesh"] = rng.choice(("2x2x2", "2x2x1", "1x2x1", "2x1x2"))
        k = more["k"] = max(k, 8)
    return {**_case(op, matrix, k, f64), **more}


_PATTERN_SEED = 1    # bench.py's default


def _operands(dev, seed, *tensors):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    for t in tensors:
        t.copy_(torch.randn(t.shape, generator=g, dtype=t.dtype, device=t.device))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    op, k = case["op"], case["k"]
    dtype = torch.float64 if case["f64"] else torch.float32
    m = generate.from_spec(case["matrix"], seed=_PATTERN_SEED)
    m.vals = np.random.default_rng(seed).random(m.nnz)
    if op == "mesh":
        return _prepare_mesh(case, m, seed, dtype, dev)
    _, plan = build_my_plan(m, Mesh3D(1, 1, 1), 0, seed=_PATTERN_SEED)
    if op == "sddmm":
        o = DistSDDMM(plan, None, k, dtype, dev)
        _operands(dev, seed, o.A_owned, o.B_owned)
        return {"run": lambda: o.run_async()}
    if op == "spmm":
        o = DistSpMM(plan, None, k, dtype, dev)
        _operands(dev, seed, o.X_owned, o.Y_owned)
        beta = case.get("beta", 0.0)
        return {"run": lambda: o.run_async(beta)}
    if op == "gat":
        layer = GatLayer(plan, None, k, dtype, dev)
        layer.sddmm.timer.enabled = layer.spmm.timer.enabled = False   # as cli.sweep times the chain: no phase timers
        _operands(dev, seed, layer.sddmm.A_owned, layer.sddmm.B_owned, layer.spmm.X_owned)
        return {"run": lambda: {"y": layer.run(), "scores": layer.spmm.vals}}
    step = SddmmSpmmStep(plan, None, k, dtype, dev, seed=seed)
    step.fill_device_operands()
    if op == "step":
        return {"run": lambda: step.run_device()}
    step.make_host_operands()
    return {"run": lambda: {"sums": step.run_e2e(), "c": step.sddmm.partial, "y": step.spmm.Y_owned}}


def _prepare_mesh(case, m, seed, dtype, dev):
    mesh, k = Mesh3D.parse(case["mesh"]), case["k"]
    _, plans = build_all_plans(m, mesh, seed=_PATTERN_SEED)
    kl = [split_k(k, mesh.Z, plans[r].coords[2])[1] for r in range(mesh.size)]
    fabric = LocalFabric(mesh.size, dev)
    keep, launches = [fabric], []
    for cls, F in ((DistSDDMM, FusedSDDMM), (DistSpMM, FusedSpMM)):
        heaps = fabric.heaps([F.region_sizes(plans[r], kl[r], dtype=dtype) for r in range(mesh.size)])
        ops = [cls(plans[r], None, k, dtype, dev, "fused", heap=heaps[r], timeout_s=5.0) for r in range(mesh.size)]
        for r, o in enumerate(ops):
            _operands(dev, seed * 64 + r, *((o.A_owned, o.B_owned) if cls is DistSDDMM else (o.X_owned, o.Y_owned)))
        keep.append(ops)
        launches.append(([o._fused for o in ops], [(o.Y_owned, 0.0) for o in ops] if cls is DistSpMM else None))

    def go():
        for fused, args in launches:
            run_lockstep(fused, args)
        return [f.out[:f.out_len] for f in launches[0][0]] + [y for y, _ in launches[1][1]]
    return {"run": go, "keep": keep}


def run(state):
    return state["run"]()


def _rmat_counts(scale, ef):
    """Expected (nonzeros without duplicates, rows that hold one) of an R-MAT graph: cells and rows are grouped by how
    often each of the four (two) branches is taken on the way down."""
    n, f = scale, math.factorial
    draws = ef * 2.0 ** scale

    def some(p):
        return -math.expm1(-draws * p)
    nnz = sum(f(n) / (f(a) * f(b) * f(c) * f(n - a - b - c)) * some(0.57 ** a * 0.19 ** (b + c) * 0.05 ** (n - a - b - c))
              for a in range(n + 1) for b in range(n + 1 - a) for c in range(n + 1 - a - b))
    rows = sum(math.comb(n, j) * some(0.76 ** (n - j) * 0.24 ** j) for j in range(n + 1))
    return nnz, rows


def _shape(matrix):
    """(nonzeros, rows, rows with a nonzero, columns with a nonzero), expected."""
    kind, *a = matrix.split(":")
    if kind == "rmat":
        nnz, used = _rmat_counts(int(a[0]), int(a[1]))
        return nnz, 1 << int(a[0]), used, used
    rows, cols = int(a[0]), int(a[1])
    if kind == "zipf":
        alpha, dmax = float(a[2]), min(int(a[3]), cols)
        nnz = rows * sum(x ** (1 - alpha) for x in range(1, dmax + 1))
    else:
        nnz = rows * float(a[2])
    used_rows = rows * -math.expm1(-float(a[2])) if kind == "er" else rows
    return nnz, rows, used_rows, cols * -math.expm1(-nnz / cols)


def work(case):
    """Column index, value and row pointer of S, every dense row that a nonzero names, and every result, once each."""
    es, k, op = (8 if case["f64"] else 4), case["k"], case["op"]
    nnz, rows, used_rows, used_cols = _shape(case["matrix"])
    layers = Mesh3D.parse(case["mesh"]).Z if op == "mesh" else 1    # every Z layer holds all of S
    sparse = (nnz * (4 + es) + 8 * rows) * layers
    sddmm = sparse + (used_rows + used_cols) * k * es + nnz * es
    spmm = sparse + (rows + used_cols) * k * es + (rows * k * es if case.get("beta") else 0)
    flops = {"sddmm": 2, "spmm": 2}.get(op, 4) * nnz * k
    return {"bytes": {"sddmm": sddmm, "spmm": spmm}.get(op, sddmm + spmm), "flops": flops}


def tolerance(case):
    """Sums of at most a few thousand products in the value type of the case, in any order.  The sums of a whole
    result that "e2e" reads back add numbers of both signs, so that the sum is smaller than what it is made of."""
    if case["f64"]:
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 5e-5 if case["op"] == "e2e" else 1e-5, "max": 1e-3}
