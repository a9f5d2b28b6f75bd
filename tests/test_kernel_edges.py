"""SDDMM and SpMM at the sizes where their split of the work changes: widths that take 16-, 8- and 4-byte vectors and
every lanes-per-row shape, lists that end inside a window or a quad, rows that cross the lane groups of an item, empty
rows, rows cut into pieces, index arrays that do not start on a 16-byte boundary.

Reference: fp64 sums of the same (already rounded) inputs.  A sum of n products in precision u, in any order, is off
by at most gamma(n) = n u / (1 - n u) times the sum of the products' magnitudes (Higham, "Accuracy and Stability of
Numerical Algorithms", section 3.1); two more roundings cover the scaling and the previous result."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def _gamma(n, dtype):
    return n * U[dtype] / (1 - n * U[dtype])


def _strided(rows, k, ld, dtype, g):
    return torch.randn(rows, ld, generator=g, dtype=torch.float64).to(dtype)[:, :k]


def _on_gpu(t, shift):
    """Copy on the GPU whose first element sits `shift` elements behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + shift, dtype=t.dtype, device="cuda")
    buf[shift:].copy_(t)
    return buf[shift:]


WIDTHS = [1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 33, 48, 50, 66, 96, 98, 100, 129, 130, 192, 200, 258, 260, 400, 512, 1024]


def _check_sddmm(rows, cols, k, dtype, shift=0, ld=None, nrows=40, ncols=50, seed=0):
    from spcomm3d_b200.ops import local
    g = torch.Generator().manual_seed(seed)
    ld = ld or k
    A, B = _strided(nrows, k, ld, dtype, g), _strided(ncols, k, ld, dtype, g)
    s = torch.rand(len(rows), generator=g, dtype=torch.float64).to(dtype)
    r, c = torch.as_tensor(rows, dtype=torch.int32), torch.as_tensor(cols, dtype=torch.int32)
    a, b = A.double()[r.long()], B.double()[c.long()]
    ref, mag = (a * b).sum(1) * s.double(), (a * b).abs().sum(1) * s.double()
    out = torch.full((len(rows),), float("nan"), dtype=dtype, device="cuda")
    Ad = torch.empty(nrows, ld, dtype=dtype, device="cuda")[:, :k]
    Bd = torch.empty(ncols, ld, dtype=dtype, device="cuda")[:, :k]
    Ad.copy_(A), Bd.copy_(B)
    local.sddmm(_on_gpu(r, shift), _on_gpu(c, shift), s.cuda(), Ad, Bd, out)
    err = (out.cpu().double() - ref).abs()
    assert bool((err <= _gamma(k + 2, dtype) * mag).all()), float((err / mag.clamp_min(1e-300)).max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", WIDTHS)
def test_sddmm_widths(dtype, k):
    rng = np.random.default_rng(k)
    rows = np.sort(rng.integers(0, 40, 301))
    _check_sddmm(rows, rng.integers(0, 50, 301), k, dtype)
    _check_sddmm(rows, rng.integers(0, 50, 301), k, dtype, shift=1, ld=k + 3)


@pytest.mark.parametrize("k", [8, 33, 64, 128])
@pytest.mark.parametrize("nnz", [1, 2, 3, 4, 5, 15, 16, 17, 31, 33, 63, 65, 127, 128, 129, 511, 513])
def test_sddmm_list_ends(k, nnz):
    rng = np.random.default_rng(nnz)
    _check_sddmm(np.sort(rng.integers(0, 40, nnz)), rng.integers(0, 50, nnz), k, torch.float32)


def _check_sddmm_places(nnz, k, dtype, place, lists=0, twice=False, runs=(1, 2, 3, 5, 6, 90)):
    """SDDMM whose values, results and second results start `place` elements behind a 16-byte boundary, the index lists
    `lists` elements."""
    from spcomm3d_b200.ops import cuda_ops
    rng = np.random.default_rng(nnz)
    deg = rng.choice(runs, nnz)
    r = torch.from_numpy(np.repeat(np.arange(deg.size), deg)[:nnz] % 40).int()
    c = torch.from_numpy(rng.integers(0, 50, nnz)).int()
    g = torch.Generator().manual_seed(k)
    A, B = _strided(40, k, k, dtype, g), _strided(50, k, k, dtype, g)
    s = torch.rand(nnz, generator=g, dtype=torch.float64).to(dtype)
    at = r.long() * 50 + c.long()
    ref = (A.double() @ B.double().T).reshape(-1)[at] * s.double()
    mag = (A.double().abs() @ B.double().abs().T).reshape(-1)[at] * s.double()
    bufs = [torch.full((nnz + 8,), float("nan"), dtype=dtype, device="cuda") for _ in range(2)]
    out, also = (b[place:place + nnz] for b in bufs)
    cuda_ops.bind_sddmm(_on_gpu(r, lists), _on_gpu(c, lists), _on_gpu(s, place), A.cuda(), B.cuda(), out,
                        also if twice else None, pack=False).launch()
    for b in bufs[:1 + twice]:
        got = b.cpu().double()
        assert bool(((got[place:place + nnz] - ref).abs() <= _gamma(k + 2, dtype) * mag).all())
        assert bool(got[:place].isnan().all()) and bool(got[place + nnz:].isnan().all())   # nothing else is written


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", [4, 16, 20, 32, 44, 64, 100, 128, 200, 256, 400, 600])   # every lanes-per-row shape
def test_sddmm_many_windows(dtype, k):
    """More windows than warps (606,208 nonzeros where a lane holds one vector), the last one short, and the lists,
    values and results at places that take no vectors."""
    _check_sddmm_places(650_003, k, dtype, 0)
    _check_sddmm_places(650_002, k, dtype, 1, lists=1, twice=True)
    _check_sddmm_places(650_001, k, dtype, 0, runs=(1,))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", [4, 33, 50, 64, 128])
@pytest.mark.parametrize("nnz", [1, 5, 130, 4097, 100_001, 420_001])
def test_sddmm_places(dtype, k, nnz):
    """One window per warp, and two or three (420,001 where a lane holds several vectors)."""
    for place, twice in ((0, True), (1, False), (2, True), (3, True)):
        _check_sddmm_places(nnz, k, dtype, place, lists=place, twice=twice)


@pytest.mark.parametrize("k", [32, 64, 128])
@pytest.mark.parametrize("nnz", [200, 700_000])   # 700,000: full windows of 128 nonzeros
def test_sddmm_row_changes(k, nnz):
    """Runs of 1, 2, 3, 4, 5 and 300 nonzeros per row; and a list that leaves a row and comes back to it."""
    rng = np.random.default_rng(7)
    runs = rng.choice([1, 1, 2, 3, 4, 5, 300], nnz)
    rows = np.repeat(np.arange(runs.size), runs)[:nnz] % 40
    _check_sddmm(rows, rng.integers(0, 50, nnz), k, torch.float32)
    again = rng.choice([3, 7], nnz)
    _check_sddmm(again, rng.integers(0, 50, nnz), k, torch.float32)


def _check_spmm(deg, k, dtype, beta, shift=0, ld=None, ncols=60, seed=0, bound_call=False, **items):
    from spcomm3d_b200.ops import cuda_ops, local
    g = torch.Generator().manual_seed(seed)
    deg = np.asarray(deg, np.int64)
    nrows, ld = deg.size, ld or k
    rowptr = torch.zeros(nrows + 1, dtype=torch.int64)
    rowptr[1:] = torch.from_numpy(np.cumsum(deg))
    nnz = int(rowptr[-1])
    ri = torch.from_numpy(np.repeat(np.arange(nrows), deg)).int()
    ci = torch.randint(0, ncols, (nnz,), generator=g).int()
    v = torch.rand(nnz, generator=g, dtype=torch.float64).to(dtype)
    X, Y0 = _strided(ncols, k, ld, dtype, g), _strided(nrows, k, ld, dtype, g)
    ref, mag = beta * Y0.double(), abs(beta) * Y0.double().abs()
    prod = X.double()[ci.long()] * v.double()[:, None]
    ref.index_add_(0, ri.long(), prod)
    mag.index_add_(0, ri.long(), prod.abs())
    Xd = torch.empty(ncols, ld, dtype=dtype, device="cuda")[:, :k]
    Xd.copy_(X)
    args = (rowptr.cuda(), ri.cuda(), _on_gpu(ci, shift), _on_gpu(v, shift), Xd)
    sched = cuda_ops.SpmmSchedule(args[0], **items)
    bound = torch.from_numpy(_gamma(deg + 3.0, dtype))[:, None] * mag
    got = []
    for _ in range(2):
        wide = torch.full((nrows, ld), 7.0, dtype=dtype, device="cuda")
        Yd = wide[:, :k]
        Yd.copy_(Y0) if beta else Yd.fill_(float("nan"))
        if bound_call:
            cuda_ops.bind_spmm(args[0], *args[2:], Yd, sched).launch(beta)
        else:
            local.spmm(*args, Yd, beta, sched)
        assert bool(((Yd.cpu().double() - ref).abs() <= bound).all())
        assert bool((wide[:, k:] == 7.0).all())
        got.append(Yd)
    assert torch.equal(got[0], got[1])          # reproducible, the counters are back at zero
    assert int(sched.counters.abs().sum()) == 0 and int(sched.ticket.abs().sum()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", WIDTHS)
def test_spmm_widths(dtype, k):
    deg = np.random.default_rng(k).poisson(6, 90)
    deg[[0, 40, 41, 89]] = 0
    deg[50] = 333                                # cut into pieces
    _check_spmm(deg, k, dtype, 0.0)
    _check_spmm(deg, k, dtype, 0.5, shift=1, ld=k + 3)


@pytest.mark.parametrize("k", [8, 32, 64, 128, 33])
@pytest.mark.parametrize("deg", [[0], [1], [3], [4], [5], [0, 0, 0], [0] * 70, [64], [65], [63, 1], [1] * 33, [1] * 64,
                                 [15, 1], [16, 16], [17, 15], [0, 16, 0, 0, 16, 0], [2, 60, 2], [5000], [64, 65, 0, 64],
                                 [130_000, 3]])
def test_spmm_items(k, deg):
    """Rows that fill, straddle and span the shares of the lane groups; rows of one item and of many pieces."""
    _check_spmm(deg, k, torch.float32, 0.0)
    _check_spmm(deg, k, torch.float32, 1.0, shift=3)


@pytest.mark.parametrize("k", [32, 128])
def test_spmm_many_items(k):
    """More items than warps: handed out dynamically, full-size items and pieces of 512."""
    rng = np.random.default_rng(3)
    deg = np.minimum(rng.zipf(1.9, 30_000), 3000)
    deg = np.concatenate([deg, np.full(8000, 90), [5000, 513, 512]])
    _check_spmm(deg, k, torch.float32, 0.5)


# Items that one round of a shape with fewer vectors per lane takes, and ones of several rows: (bytes of a row) / 16 from
# 11 to 64, both sides of 17, 25, 33 and 49.
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nvec", [11, 16, 17, 24, 25, 32, 33, 48, 49, 64])
def test_spmm_one_round(dtype, nvec):
    k = nvec * 16 // (4 if dtype == torch.float32 else 8)
    rows = 4375 if nvec <= 32 else 2500
    _check_spmm([16] * rows, k, dtype, 0.5 if nvec % 2 else 0.0, bound_call=True)
    _check_spmm([4] * rows, k, dtype, 0.0, bound_call=True, item_nnz=4)
    _check_spmm([16] * rows, k, dtype, 0.5)
    _check_spmm([16] * 3000, k, dtype, 0.0)
    _check_spmm([6, 7] * 900, k, dtype, 0.5, bound_call=True)
    _check_spmm([16] * 4000 + [90], k, dtype, 0.0, bound_call=True)    # one split row


@pytest.mark.parametrize("k", [8, 20, 64, 96, 128, 256])
def test_spmm_longest_items(k):
    """Items of 256 nonzeros, which matrices of more than six million take: one row, 32 short ones, and pieces of 512."""
    _check_spmm([8] * 70 + [300, 1, 511] + [0] * 40 + [513, 1400] + [37] * 20, k, torch.float32, 0.5, item_nnz=256, long_row=512)
    _check_spmm([256] * 9 + [255, 257, 1] * 3, k, torch.float64, 0.0, item_nnz=256, long_row=512)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("gen,k", [("uniform:5:7:3", 3), ("er:70001:50000:3", 33), ("zipf:40000:90000:1.8:300", 64)])
def test_step_from_host_operands(dtype, gen, k):
    """The step queued by one native call (operands in one part and in several) leaves what the two operators leave
    when they are run one after the other on the same operands, and returns the sums of it."""
    from spcomm3d_b200.models.layer import SddmmSpmmStep
    from spcomm3d_b200.parallel.mesh import Mesh3D
    from spcomm3d_b200.parallel.plan import build_my_plan
    from spcomm3d_b200.utils import generate
    m = generate.from_spec(gen, seed=4)
    _, plan = build_my_plan(m, Mesh3D(1, 1, 1), 0, seed=4)
    step = SddmmSpmmStep(plan, None, k, dtype, "cuda", seed=2)
    step.fill_device_operands()
    c, y = (t.clone() for t in step.run_device())
    step.make_host_operands()
    for t in (step.sddmm.A_owned, step.sddmm.B_owned, step.spmm.X_owned, step.sddmm.partial, step.spmm.Y_owned):
        t.fill_(7.0)
    for _ in range(2):
        sums = step.run_e2e()
    assert torch.equal(step.sddmm.run_async(), c) and torch.equal(step.spmm.Y_owned, y)
    # the checksum adds fp64 values in a fixed shape; torch adds them in another: both within n u of the magnitudes
    for got, t in zip(sums, (c, y)):
        t = t.double()
        assert abs(got - float(t.sum())) <= 2 * t.numel() * 2.0 ** -53 * float(t.abs().sum())
    step.host = {"A": step.host["A"] * 2, "B": step.host["B"] * 2}      # operands of the user's own
    twice = step.run_e2e()
    assert twice[1] == 2 * sums[1] and twice[0] == 4 * sums[0]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k, n", [(12, 1), (13, 5), (33, 259), (64, 3001), (128, 130), (200, 2048), (512, 77)])
def test_sddmm_column_chunks(dtype, k, n, monkeypatch):
    """Columns chunk by chunk: the values stay in row order and are those of the row-sorted lists, bit for bit (a dot
    product is computed by the same lanes in either order), through the operator too."""
    from spcomm3d_b200.models.dist_ops import DistSDDMM
    from spcomm3d_b200.ops import cuda_ops, local
    from spcomm3d_b200.parallel.mesh import Mesh3D
    from spcomm3d_b200.parallel.plan import build_my_plan
    from spcomm3d_b200.utils.sparse import CooMatrix
    rng = np.random.default_rng(n)
    keys = np.sort(rng.choice(60 * 64, n, replace=False))
    m = CooMatrix(60, 64, (keys // 64).astype(np.int32), (keys % 64).astype(np.int32), rng.random(n))
    _, plan = build_my_plan(m, Mesh3D(1, 1, 1), 0, seed=1)
    chosen = []

    def chunks(r, c, n_cols, row_bytes, _f=cuda_ops.column_chunks):
        chosen.append(_f(r, c, n_cols, row_bytes, force=5))
        return chosen[-1]
    monkeypatch.setattr(cuda_ops, "column_chunks", chunks)
    op = DistSDDMM(plan, None, k, dtype, "cuda")
    assert chosen and op._chunks is chosen[0]
    for t, stream in ((op.A_owned, 1), (op.B_owned, 2)):
        t.copy_(torch.randn(t.shape, generator=torch.Generator().manual_seed(stream), dtype=torch.float64))
    ref = torch.empty_like(op.partial)
    local.sddmm(op.rowidx, op.colidx, op.vals, op._A_full, op._B_full, ref)
    op.partial.fill_(float("nan"))
    assert torch.equal(op.run_async(), ref)
    op.partial.fill_(float("nan"))
    assert torch.equal(op.run(), ref)


def test_column_chunks_rule(monkeypatch):
    """Chunks where every column is read equally often from a B larger than the limit, none where hub columns or the
    size of B leave nothing to gain."""
    from spcomm3d_b200.ops import cuda_ops
    monkeypatch.setattr(cuda_ops, "CHUNK_BYTES", 1 << 18)
    monkeypatch.setattr(cuda_ops, "CHUNK_MIN_NNZ", 1)
    rng = np.random.default_rng(0)
    rows = torch.arange(4096, dtype=torch.int32).repeat_interleave(64).cuda()

    def lists(cols):
        return rows, torch.from_numpy(np.sort(cols, 1).astype(np.int32)).reshape(-1).cuda()
    even = lists(rng.integers(0, 4096, (4096, 64)))
    r, c, where = cuda_ops.column_chunks(*even, 4096, 256)
    assert torch.equal(r[where.long()], even[0]) and torch.equal(c[where.long()], even[1])
    assert bool((torch.diff(c // 1024) >= 0).all()) and torch.unique(where).numel() == where.numel()
    assert cuda_ops.column_chunks(*even, 4096, 48) is None      # fits
    hubs = lists(np.where(rng.random((4096, 64)) < 0.8, rng.integers(0, 512, (4096, 64)), rng.integers(0, 4096, (4096, 64))))
    assert cuda_ops.column_chunks(*hubs, 4096, 256) is None


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", [32, 44, 64, 100, 128, 200, 256, 400])   # every number of vectors per lane
def test_rows_shorter_than_quads(dtype, k):
    """Rows of one nonzero and more: quads of one to four rows (SDDMM), several row ends in a quad, in every quad of a
    group and at its last position, and one long row alone (SpMM)."""
    for run in ([1], [2], [3], [4], [5], [1, 3], [2, 1, 1], [1, 2, 7, 40], [4, 4, 1, 300]):
        deg = (run * 40)[:40]
        rows = np.repeat(np.arange(40), deg)
        _check_sddmm(rows, np.random.default_rng(len(rows)).integers(0, 50, len(rows)), k, dtype)
        _check_spmm(deg, k, dtype, 0.0)
        _check_spmm(deg, k, dtype, 0.5, shift=1)
    _check_spmm([130], k, dtype, 0.5)
    _check_spmm([0, 511, 0, 512], k, dtype, 0.0)
