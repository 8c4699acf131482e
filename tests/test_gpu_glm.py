"""GPU numerics of the GLM kernels against plain PyTorch fp32/fp64 references."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _random_csr(rows, dim, nnz_lo, nnz_hi, seed, binary=False, zipf=True):
    from sketchml_b200.data import CSRMatrix
    rng = np.random.default_rng(seed)
    counts = rng.integers(nnz_lo, nnz_hi + 1, rows)
    rowptr = np.zeros(rows + 1, np.int64)
    rowptr[1:] = np.cumsum(counts)
    cols = np.empty(rowptr[-1], np.int32)
    for r in range(rows):
        if zipf:
            p = 1.0 / np.arange(1, dim + 1) ** 1.1
            c = rng.choice(dim, counts[r], replace=False, p=p / p.sum())
        else:
            c = rng.choice(dim, counts[r], replace=False)
        cols[rowptr[r]:rowptr[r + 1]] = np.sort(c)
    vals = None if binary else torch.from_numpy(rng.normal(size=rowptr[-1]).astype(np.float32))
    labels = torch.from_numpy(np.where(rng.random(rows) < 0.5, 1.0, -1.0).astype(np.float32))
    return CSRMatrix(torch.from_numpy(rowptr), torch.from_numpy(cols), vals, labels, dim)


def _ref_grad(m, w, loss, lo, hi, lam):
    b = m.slice_rows(lo, hi)
    w64 = w.double().cpu()
    pre = loss.predict(w64, b)
    y = b.labels.double()
    coef = -loss.grad(pre, y) / (hi - lo)
    g = torch.zeros(m.dim, dtype=torch.float64)
    g.index_add_(0, b.cols.long(), coef[b.row_ids()] * b.dense_values(torch.float64))
    touched = g.abs() > 0
    full = g + lam * w64 * touched
    keep = touched & (full.abs() > 1e-8)
    return full, keep, float(loss.loss(pre, y).sum())


@pytest.mark.parametrize("loss_name,binary,nnz", [("log", True, (20, 20)), ("hinge", False, (1, 70)), ("square", False, (150, 260))])
def test_grad_compact_matches_reference(loss_name, binary, nnz):
    from sketchml_b200.models.loss import L2HingeLoss, L2LogLoss, L2SquareLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    dev = torch.device("cuda")
    loss = {"log": L2LogLoss, "hinge": L2HingeLoss, "square": L2SquareLoss}[loss_name](1e-3)
    dim, rows = 20000, 700
    m = _random_csr(rows, dim, nnz[0], nnz[1], seed=nnz[0], binary=binary)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim) * 0.3).float()
    wd = w.to(dev)
    st = GlmState.create(dim, dim, dev)
    lo, hi = 37, 650
    st.partials.zero_()
    glm_grad(csr, [(lo, hi)], wd, st, loss.loss_id, hi - lo, hot=4096)
    compact_gradient(st, wd, loss.lam)
    torch.cuda.synchronize()
    assert int(st.status.item()) == 0
    n = int(st.meta[0])
    keys = st.keys[:n].cpu().long()
    vals = st.vals[:n].cpu().double()
    full, keep, ref_loss = _ref_grad(m, w, loss, lo, hi, loss.lam)
    ref_keys = torch.nonzero(keep).flatten()
    # coordinates whose magnitude sits at the 1e-8 filter may differ; compare as dense vectors
    got = torch.zeros(dim, dtype=torch.float64)
    got[keys] = vals
    ref = torch.where(keep, full, torch.zeros_like(full))
    assert torch.all(keys[1:] > keys[:-1])
    assert abs(n - ref_keys.numel()) <= max(2, ref_keys.numel() // 1000)
    scale = float(ref.abs().max())
    assert float((got - ref).abs().max()) <= 2e-5 * max(scale, 1.0) + 1e-7
    assert abs(float(st.partials[1]) - ref_loss) <= 1e-3 * max(1.0, abs(ref_loss))
    # accumulator and bitmap are clean for the next step
    assert float(st.g.abs().max()) == 0.0 and int(st.bitmap.abs().max()) == 0


def test_wraparound_segments_and_validation():
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad, glm_validate
    from sketchml_b200.trainer import validation_counts
    dev = torch.device("cuda")
    loss = L2LogLoss(0.0)
    dim, rows = 5000, 300
    m = _random_csr(rows, dim, 5, 40, seed=3)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim) * 0.5).float()
    wd = w.to(dev)
    st = GlmState.create(dim, dim, dev)
    st.partials.zero_()
    glm_grad(csr, [(250, 300), (0, 70)], wd, st, loss.loss_id, 120, hot=1024)
    compact_gradient(st, wd, 0.0)
    n = int(st.meta[0])
    got = torch.zeros(dim, dtype=torch.float64)
    got[st.keys[:n].cpu().long()] = st.vals[:n].cpu().double()
    f1, k1, _ = _ref_grad(m, w, loss, 250, 300, 0.0)
    f2, k2, _ = _ref_grad(m, w, loss, 0, 70, 0.0)
    ref = f1 * 50 / 120 + f2 * 70 / 120
    ref = torch.where(ref.abs() > 1e-8, ref, torch.zeros_like(ref))
    assert float((got - ref).abs().max()) < 1e-5
    acc = glm_validate(csr, wd, loss.loss_id, st.status).cpu()
    pre = loss.predict(w.double(), m)
    refc = validation_counts(pre, m.labels.double(), loss)
    assert abs(acc[0] - refc[0]) < 1e-3 * refc[0]
    assert [int(x) for x in acc[1:6]] == [int(x) for x in refc[1:6]]


def test_dense_kind_decision_and_values():
    from sketchml_b200.models.loss import L2SquareLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    dev = torch.device("cuda")
    loss = L2SquareLoss(1e-2)
    dim, rows = 600, 200
    m = _random_csr(rows, dim, 100, 200, seed=9, zipf=False)
    csr = DeviceCSR(m, dev)
    w = torch.randn(dim).float()
    wd = w.to(dev)
    st = GlmState.create(dim, dim, dev, allow_dense=True)
    st.partials.zero_()
    glm_grad(csr, [(0, rows)], wd, st, loss.loss_id, rows, hot=256)
    compact_gradient(st, wd, loss.lam)
    assert int(st.meta[1]) == 2
    full, keep, _ = _ref_grad(m, w, loss, 0, rows, 0.0)
    ref = full + loss.lam * w.double()
    assert float((st.dense_vals.cpu().double() - ref).abs().max()) < 1e-4 * float(ref.abs().max())


def test_device_generator_statistics():
    from sketchml_b200.data.synthetic import SyntheticSpec, zipf_inverse_cdf
    from sketchml_b200.ops import generate_gpu
    spec = SyntheticSpec(rows=20000, dim=100000, nnz_per_row=20, zipf_s=1.1, values="binary", task="logistic", seed=5)
    csr, w = generate_gpu(spec, 0, spec.rows, "cuda")
    cols = csr.cols[:csr.nnz].cpu().numpy().reshape(spec.rows, 20)
    assert cols.min() >= 0 and cols.max() < spec.dim
    srt = np.sort(cols, axis=1)
    assert (srt[:, 1:] != srt[:, :-1]).all(), "columns repeat inside a row"
    # head mass of the Zipf law: column 0 is in most rows, and rank frequencies decay
    f0 = (cols == 0).any(axis=1).mean()
    exp = zipf_inverse_cdf(np.random.default_rng(0).random(400000), spec.dim, 1.1)
    p0 = (exp == 0).mean()
    assert abs(f0 - (1 - (1 - p0) ** 20)) < 0.08
    lab = csr.labels.cpu().numpy()
    assert set(np.unique(lab)) <= {-1.0, 1.0} and 0.2 < (lab > 0).mean() < 0.8
    wn = w.cpu().numpy()
    assert abs((wn != 0).mean() - 0.1) < 0.01
    spec2 = SyntheticSpec(rows=2000, dim=5000, nnz_per_row=200, zipf_s=0.0, values="uniform_l2", task="svm", seed=6)
    c2, _ = generate_gpu(spec2, 100, 2000, "cuda")
    v = c2.values[:c2.nnz].cpu().numpy().reshape(2000, 200)
    assert np.allclose((v ** 2).sum(axis=1), 1.0, atol=1e-4)


@pytest.mark.parametrize("binary", [True, False])
def test_transposed_index_gradient_matches_scatter_path(binary):
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    from sketchml_b200.ops.transposed import build_batch_index, glm_grad_transposed
    dev = torch.device("cuda")
    loss = L2LogLoss(1e-3)
    dim, rows = 30000, 6000
    m = _random_csr(rows, dim, 1, 60, seed=21, binary=binary)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim) * 0.3).float().to(dev)
    st = GlmState.create(dim, dim, dev)
    lo, hi = 2000, 4000
    st.partials.zero_()
    glm_grad(csr, [(lo, hi)], w, st, loss.loss_id, hi - lo, hot=2048)
    compact_gradient(st, w, loss.lam)
    n = int(st.meta[0])
    ref = torch.zeros(dim, dtype=torch.float64)
    ref[st.keys[:n].cpu().long()] = st.vals[:n].cpu().double()
    ref_loss = float(st.partials[1])
    bi = build_batch_index(csr, lo, hi)
    assert bi.n_short + bi.n_medium + len(torch.unique(bi.long_col)) == bi.n_cols
    assert torch.all(bi.ucols[1:] > bi.ucols[:-1]) and int(bi.colptr[-1]) == int(csr.rowptr[hi] - csr.rowptr[lo])
    coef = torch.zeros(hi - lo, device=dev)
    out = torch.zeros(dim, device=dev)
    st.partials.zero_()
    glm_grad_transposed(csr, bi, w, coef, out, st.partials, st.status, loss.loss_id, loss.lam)
    got = torch.zeros(dim, dtype=torch.float64)
    got[bi.ucols.cpu().long()] = out[:bi.n_cols].cpu().double()
    assert int(st.status.item()) == 0
    assert abs(float(st.partials[1]) - ref_loss) < 1e-3 * abs(ref_loss)
    assert abs(bi.n_cols - n) <= 3          # the scatter path drops |v| <= 1e-8, this one keeps them
    assert float((got - ref).abs().max()) < 2e-6 * max(1.0, float(ref.abs().max())) + 2e-8


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("tile_rows_max,rows", [(49152, 2000), (512, 2000), (1000, 5003), (49152, 60000)])
def test_row_tiled_index_matches_the_per_column_form(binary, tile_rows_max, rows, monkeypatch):
    """The row-tiled index (tile coefficients in shared memory, partial sums per (tile, column) pair added in
    tile order) gives the gradient of the per-column form up to the order of the float adds, the same keys,
    and the same bits on every repetition."""
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR, GlmState
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", tile_rows_max)
    dev = torch.device("cuda")
    loss = L2LogLoss(1e-3)
    dim = 30000
    m = _random_csr(rows + 500, dim, 1, 40, seed=33, binary=binary)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim) * 0.3).float().to(dev)
    st = GlmState.create(dim, dim, dev)
    lo, hi = 250, 250 + rows
    plain, tiled = T.build_batch_index(csr, lo, hi), T.build_batch_index(csr, lo, hi, tiled=True)
    assert tiled.tiled is not None and tiled.tiled.n_tiles == -(-rows // tile_rows_max)
    assert torch.equal(plain.ucols, tiled.ucols) and int(tiled.tiled.pair_ptr[-1]) == int(csr.rowptr[hi] - csr.rowptr[lo])
    assert int(tiled.tiled.col_pair_ptr[-1]) == tiled.tiled.n_pairs
    coef = torch.zeros((rows + 3) // 4 * 4, device=dev)
    outs = []
    for bi in (plain, tiled, tiled):
        out = torch.full((dim,), 7.0, device=dev)
        st.partials.zero_()
        T.glm_grad_transposed(csr, bi, w, coef, out, st.partials, st.status, loss.loss_id, loss.lam)
        assert int(st.status.item()) == 0
        outs.append(out[:bi.n_cols].clone())
    assert torch.equal(outs[1], outs[2])
    assert float((outs[0].double() - outs[1].double()).abs().max()) < 2e-6 * max(1.0, float(outs[0].abs().max()))



@pytest.mark.parametrize("dim", [1, 31, 33, 256, 257, 8 * 256 + 1, 100_000, 4096 * 256, 4096 * 256 + 1, 3_000_001])
@pytest.mark.parametrize("density", [0.02, 0.6, 0.95])
def test_compaction_over_its_splits(dim, density):
    """Edges of the warps' word ranges: one warp, a ragged last warp, the last size with the smallest range and the
    first with the next one; sparse words, dense words and the dense kind."""
    from sketchml_b200.ops.glm import GlmState, compact_gradient
    dev, lam = torch.device("cuda"), 0.5
    gen = torch.Generator().manual_seed(dim)
    touched = torch.rand(dim, generator=gen) < density
    g = torch.where(touched, torch.randn(dim, generator=gen), torch.zeros(dim))
    g[::9] = torch.where(touched[::9], torch.full_like(g[::9], 1e-9), g[::9])   # falls to the filter where w is zero
    w = torch.randn(dim, generator=gen)
    w[::9] = 0.0
    for allow_dense in (False, True):
        st = GlmState.create(dim, dim, dev, allow_dense)
        st.g.copy_(g)
        words = torch.zeros((dim + 31) // 32 * 32, dtype=torch.int64)
        words[:dim] = touched.long()
        bits = (words.view(-1, 32) << torch.arange(32)).sum(1)
        st.bitmap[:bits.numel()].copy_(torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits).to(torch.int32))
        compact_gradient(st, w.to(dev), lam)
        v = (g + lam * w)    # one rounding of the product, one of the sum (or a fused one): 2 ulp
        keep = touched & (v.abs() > 1e-8)
        n, kind = int(st.meta[0]), int(st.meta[1])
        assert int(st.status.item()) == 0 and n == int(keep.sum())
        dense = allow_dense and n > dim * 2 // 3
        assert kind == (0 if n == 0 else 2 if dense else 1)
        if dense:
            want = torch.where(touched & ~keep, torch.zeros(dim), torch.where(keep, v, lam * w))
            want = torch.where(touched & ~keep, lam * w, want)
            assert torch.allclose(st.dense_vals.cpu(), want, rtol=3e-7, atol=3e-7)
        else:
            idx = torch.nonzero(keep).flatten()
            assert torch.equal(st.keys[:n].cpu().long(), idx)
            assert torch.allclose(st.vals[:n].cpu(), v[idx], rtol=3e-7, atol=3e-7)
        assert float(st.g.abs().max()) == 0.0 and int(st.bitmap.abs().max()) == 0


@pytest.mark.parametrize("rows", [1, 3, 31, 33, 1000, 30011])
@pytest.mark.parametrize("nnz", [(0, 5), (1, 30), (20, 60), (90, 300)])
@pytest.mark.parametrize("binary", [True, False])
def test_margins_over_their_row_shapes(rows, nnz, binary):
    """Lanes per row (by the average length), turns per warp (by the row count), empty rows, rows longer than a trip,
    columns on both sides of the ones kept in shared memory: coefficients, loss and counts against fp64."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR, glm_validate
    from sketchml_b200.ops import lib as L
    dev, dim = torch.device("cuda"), 20000
    gen = torch.Generator().manual_seed(rows + nnz[1])
    cnt = torch.randint(nnz[0], nnz[1] + 1, (rows,), generator=gen)
    rowptr = torch.zeros(rows + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(cnt, 0)
    n = int(rowptr[-1])
    cols = (torch.rand(n, generator=gen) ** 4 * dim).int().clamp_max(dim - 1)   # frequent low columns; repeats do no harm here
    vals = None if binary else torch.randn(n, generator=gen)
    labels = torch.where(torch.rand(rows, generator=gen) < 0.5, -1.0, 1.0)
    m = CSRMatrix(rowptr, cols, vals, labels, dim)
    w = torch.randn(dim, generator=gen) * 0.2
    csr, wd = DeviceCSR(m, dev), w.to(dev)
    loss = L2LogLoss(0.0)
    pre = loss.predict(w.double(), m)
    # a margin is a sum of k <= 300 fp32 products in some order: error <= k eps sum |products| <= 300 * 6e-8 * (300 * 4)
    # in the worst case; the bound below takes the batch's largest row sum of |products|
    prod = w.abs().double()[cols.long()] * (1.0 if binary else vals.abs().double())
    row_abs = torch.zeros(rows, dtype=torch.float64).index_add_(0, torch.repeat_interleave(torch.arange(rows), cnt), prod)
    tol = 300 * 6e-8 * float(row_abs.max()) + 1e-6
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    out = torch.empty(rows, device=dev)
    acc = glm_validate(csr, wd, loss.loss_id, status, margins=out).cpu()
    assert float((out.cpu().double() - pre).abs().max()) <= tol
    assert abs(float(acc[0]) - float(loss.loss(pre, labels.double()).sum())) <= (tol + 1e-5) * rows
    assert float(acc[1] + acc[2] + acc[3] + acc[4]) == rows - int((out == 0).sum()) and float(acc[5]) == rows
    lo = min(rows - 1, 7)    # a batch that starts inside the shard
    coef = torch.empty(rows, device=dev)
    part = torch.zeros(1, dtype=torch.float64, device=dev)
    L.check(L.lib().skml_glm_coef(L.ptr(csr.rowptr), L.ptr(csr.cols), L.ptr(csr.values), L.ptr(csr.labels), lo, rows - lo,
                                  csr.nnz_padded, float(csr.avg_nnz), L.ptr(wd), dim, loss.loss_id, 0.5, L.ptr(part), L.ptr(coef),
                                  L.ptr(status), L.budget_cycles(1.0), L.stream()), "coef")
    want = -0.5 * loss.grad(pre, labels.double())[lo:]
    assert float((coef[:rows - lo].cpu().double() - want).abs().max()) <= tol + 1e-6    # slope <= 1/4; __expf: a few ulp
    assert abs(float(part) - float(loss.loss(pre, labels.double())[lo:].sum())) <= (tol + 1e-5) * rows


@pytest.mark.parametrize("rows,dim,nnz,tile", [
    (1, 40, 40, 49152), (33, 300, (250, 300), 49152), (2000, 5000, (20, 90), 49152), (2000, 5000, (20, 90), 256),
    (50000, 700, (10, 30), 49152), (3001, 1003, (60, 200), 1000)])
@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("zipf", [True, False])
def test_near_dense_index_matches_the_scatter_path(rows, dim, nnz, tile, binary, zipf, monkeypatch):
    """Tiled lists of a near-dense batch: one tile and several, ragged last tiles, lists of no entry, of a few quads
    and longer than a warp sums at once (frequent columns), margins with and without the tiled form; the batch starts
    inside the shard."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.models.loss import L2SquareLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", tile)
    dev, loss = torch.device("cuda"), L2SquareLoss(1e-2)
    gen = torch.Generator().manual_seed(rows + dim)
    lead = 5
    lo_n, hi_n = nnz if isinstance(nnz, tuple) else (nnz, nnz)
    cnt = torch.randint(lo_n, hi_n + 1, (rows + lead,), generator=gen)
    rowptr = torch.zeros(rows + lead + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(cnt, 0)
    n = int(rowptr[-1])
    u = torch.rand(n, generator=gen)
    cols = ((u ** 3 if zipf else u) * dim).int().clamp_max(dim - 1)   # a column may repeat in a row: its products just add up
    vals = None if binary else torch.randn(n, generator=gen)
    m = CSRMatrix(rowptr, cols, vals, torch.randn(rows + lead, generator=gen), dim)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim, generator=gen) * 0.1).to(dev)
    di = T.build_dense_index(csr, lead, rows + lead)
    distinct = int(torch.unique(cols[int(rowptr[lead]):]).numel())
    short = int(rowptr[-1] - rowptr[lead]) < T._tiles(rows, tile)[0] * dim
    assert (di is None) == (short or distinct <= dim * 2 // 3)
    if di is None:
        return
    st = GlmState.create(dim, dim, dev, allow_dense=True)
    di.bind(torch.empty(di.partial_floats, device=dev), torch.empty(rows, device=dev))
    T.glm_grad_dense(csr, di, w, st.g, st.bitmap, st.partials, st.status, loss.loss_id)
    # fp64 gradient; a margin sums k products in fp32, a column up to n of them: error <= 2 k eps sum |products|
    c64, e0 = cols.long(), int(rowptr[lead])
    x = (torch.ones(n) if binary else vals).double()
    rid = torch.repeat_interleave(torch.arange(rows + lead), cnt)
    pre = torch.zeros(rows + lead, dtype=torch.float64).index_add_(0, rid, w.cpu().double()[c64] * x)
    coef = (pre - m.labels.double()) / rows
    want = torch.zeros(dim, dtype=torch.float64).index_add_(0, c64[e0:], coef[rid[e0:]] * x[e0:])
    mag = torch.zeros(dim, dtype=torch.float64).index_add_(0, c64[e0:], coef[rid[e0:]].abs() * x[e0:].abs())
    row_abs = torch.zeros(rows + lead, dtype=torch.float64).index_add_(0, rid, (w.cpu().double()[c64] * x).abs())
    col_abs = torch.zeros(dim, dtype=torch.float64).index_add_(0, c64[e0:], x[e0:].abs())
    eps = 6e-8
    tol = 2 * eps * (torch.bincount(c64, minlength=dim).double().sqrt() + 20) * mag + 2 * eps * hi_n * float(row_abs.max()) / rows * col_abs + 1e-12
    assert bool(((st.g.cpu().double() - want).abs() <= tol).all())
    want_loss = 0.5 * (pre - m.labels.double())[lead:].square().sum()
    assert abs(float(st.partials[1]) - float(want_loss)) <= 1e-5 * float(want_loss)
    seen = torch.zeros(dim, dtype=torch.bool)
    seen[c64[e0:]] = True
    words = st.bitmap.cpu().long() & 0xFFFFFFFF
    got = ((words[:, None] >> torch.arange(32)) & 1).flatten()[:dim].bool()
    assert torch.equal(got, seen)
    compact_gradient(st, w, loss.lam)
    kinds = [int(st.meta[0]), int(st.meta[1])]
    assert float(st.g.abs().max()) == 0.0 and int(st.bitmap.abs().max()) == 0
    glm_grad(csr, [(lead, rows + lead)], w, st, loss.loss_id, rows, hot=256)
    compact_gradient(st, w, loss.lam)
    assert kinds == [int(st.meta[0]), int(st.meta[1])] and int(st.status.item()) == 0


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("hot", [0, 32, 8192])
@pytest.mark.parametrize("rows,nnz,dim", [(1, (1, 1), 64), (3, (0, 5), 400), (33, (0, 40), 3000), (700, (90, 300), 9001),
                                          (5000, (0, 45), 9001)])
def test_scatter_gradient_is_exact_on_whole_numbers(rows, nnz, dim, hot, binary):
    """Square loss on weights, values and labels of -1, 0, 1: every sum is a whole number below 2^24, so fp32 adds in
    any order give the fp64 gradient itself. Empty rows, rows longer than a warp, ragged last turns, no shared columns,
    private ones only, and more than the batch is worth."""
    from sketchml_b200.models.loss import L2SquareLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    rng = np.random.default_rng(rows)
    m = _random_csr(rows, dim, nnz[0], nnz[1], seed=rows + 1, binary=True, zipf=False)
    if not binary:
        m.values = torch.from_numpy(rng.integers(-1, 2, m.cols.numel()).astype(np.float32))
    x = torch.ones(m.cols.numel(), dtype=torch.float64) if binary else m.values.double()
    w = torch.from_numpy(rng.integers(-1, 2, dim).astype(np.float32))
    dev = torch.device("cuda")
    st = GlmState.create(dim, dim, dev)
    st.partials.zero_()
    loss = L2SquareLoss(0.0)
    glm_grad(DeviceCSR(m, dev), [(0, rows)], w.to(dev), st, loss.loss_id, 1, hot=hot)
    rid = torch.repeat_interleave(torch.arange(rows), m.rowptr[1:] - m.rowptr[:-1])
    pre = torch.zeros(rows, dtype=torch.float64).index_add_(0, rid, w.double()[m.cols.long()] * x)
    want = torch.zeros(dim, dtype=torch.float64).index_add_(0, m.cols.long(), (pre - m.labels.double())[rid] * x)
    assert torch.equal(st.g.cpu().double(), want)
    assert float(st.partials[1]) == float(0.5 * (pre - m.labels.double()).square().sum())
    compact_gradient(st, w.to(dev), 0.0)
    n = int(st.meta[0])
    assert torch.equal(st.keys[:n].cpu().long(), torch.nonzero(want).flatten())
    assert torch.equal(st.vals[:n].cpu().double(), want[want != 0])
    assert float(st.g.abs().max()) == 0.0 and int(st.bitmap.abs().max()) == 0 and int(st.status.item()) == 0


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("rows,dim,nnz", [(20000, 200000, 12), (3001, 20003, 90)])
def test_near_dense_index_stays_within_its_budget(rows, dim, nnz, binary):
    """Building it takes no more memory than it was allowed, scratch of a step included; where that is not enough there
    is no index. Lists of one entry, which padding makes four times as long, and lists for the margins too."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.ops import DeviceCSR
    from sketchml_b200.ops import transposed as T
    dev = torch.device("cuda")
    gen = torch.Generator().manual_seed(rows)
    cols = torch.randint(0, dim, (rows * nnz,), generator=gen).int()
    m = CSRMatrix(torch.arange(rows + 1) * nnz, cols, None if binary else torch.randn(rows * nnz, generator=gen), torch.ones(rows), dim)
    csr = DeviceCSR(m, dev)

    def build(budget):
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        di = T.build_dense_index(csr, 0, rows, budget)
        scratch = None if di is None else torch.empty(di.partial_floats, device=dev)
        torch.cuda.synchronize()
        del scratch
        return di, torch.cuda.max_memory_allocated() - before

    di, peak = build(None)
    assert di is not None and di.nbytes() <= peak
    used = di.nbytes()
    del di
    lo, hi = used // 2, 4 * peak
    while hi - lo > 65536:       # the smallest budget that is enough: what was allowed is never exceeded on the way
        mid = (lo + hi) // 2
        di, peak = build(mid)
        assert peak <= mid + 65536        # (the allocator rounds small tensors up)
        lo, hi = (lo, mid) if di is not None else (mid, hi)
        del di
    assert hi <= 4 * used


def test_near_dense_shard_without_room_for_the_index_trains_with_the_scatter(monkeypatch):
    """Ten binary batches whose lists hold one or two entries, which padding makes four: the index of all batches does
    not fit what is free, so there is none, and the steps take the scatter path."""
    from sketchml_b200.config import MLConf
    from sketchml_b200.trainer import Trainer
    free = 25_000_000
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a, **k: (free, free))
    t = Trainer(MLConf(algo="linreg", format="synthetic", feature_num=200_000, syn_rows=200_000, syn_nnz_per_row=12, syn_zipf_s=0.0,
                       syn_values="binary", valid_ratio=0.0, epoch_num=1, batch_sample_ratio=0.1, learn_rate=0.05, device="cuda"))
    t.load_data()
    assert t.engine.tindex is None or t.engine.index_bytes <= 0.8 * free
    w = t.model.weights.clone()
    t.train_one_iteration(0, 0)
    t.engine.check()
    assert not torch.equal(w, t.model.weights)
    t.close()


@pytest.mark.parametrize("loss_name,scale", [("hinge", 1.0), ("log", 60.0)])
@pytest.mark.parametrize("rows,dim,nnz,tile", [(2000, 5000, (20, 90), 49152), (2000, 5000, (20, 90), 256), (50000, 700, (10, 30), 49152),
                                               (3001, 1003, (60, 200), 1000)])
@pytest.mark.parametrize("binary", [True, False])
def test_near_dense_index_touches_the_columns_the_scatter_touches(rows, dim, nnz, tile, binary, loss_name, scale, monkeypatch):
    """Rows without a coefficient (outside the hinge, or a logistic slope that underflows) touch no column: the same
    touched bits, count and kind as the scatter's, also where a column's sum cancels. Whole-numbered weights and values
    make every margin exact; columns in no list, in short lists and in lists that a warp sums at a time."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.models.loss import L2HingeLoss, L2LogLoss
    from sketchml_b200.ops import DeviceCSR, GlmState, compact_gradient, glm_grad
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", tile)
    dev, loss = torch.device("cuda"), (L2HingeLoss if loss_name == "hinge" else L2LogLoss)(1e-3)
    gen = torch.Generator().manual_seed(rows + dim)
    cnt = torch.randint(nnz[0], nnz[1] + 1, (rows,), generator=gen)
    rowptr = torch.zeros(rows + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(cnt, 0)
    n = int(rowptr[-1])
    cols = (torch.rand(n, generator=gen) ** (1 if tile == 1000 else 1.3) * dim).int().clamp_max(dim - 1)
    vals = None if binary else torch.randint(0, 2, (n,), generator=gen).float() * 2 - 1
    w = (torch.randint(-1, 2, (dim,), generator=gen) * scale).float()
    rid = torch.repeat_interleave(torch.arange(rows), cnt)
    pre = torch.zeros(rows, dtype=torch.float64).index_add_(0, rid, (w.double()[cols.long()] * (1.0 if binary else vals.double())))
    labels = torch.where(pre > 0, 1.0, -1.0)
    few = torch.randperm(rows, generator=gen)[:max(2, dim // (nnz[0] + nnz[1]))]
    labels[few] = -labels[few]     # rows on the wrong side: with the ones near the border, those that have a coefficient
    csr = DeviceCSR(CSRMatrix(rowptr, cols, vals, labels.float(), dim), dev)
    di = T.build_dense_index(csr, 0, rows)
    if di is None:
        assert int(torch.unique(cols).numel()) <= dim * 2 // 3 or n < T._tiles(rows, tile)[0] * dim
        return
    wd, got = w.to(dev), []
    for form in ("index", "scatter"):
        st = GlmState.create(dim, dim, dev, allow_dense=True)
        if form == "index":
            di.bind(torch.empty(di.partial_floats, device=dev), torch.empty(rows, device=dev))
            T.glm_grad_dense(csr, di, wd, st.g, st.bitmap, st.partials, st.status, loss.loss_id)
        else:
            glm_grad(csr, [(0, rows)], wd, st, loss.loss_id, rows, hot=0)
        bitmap = st.bitmap.clone()
        compact_gradient(st, wd, loss.lam)
        got.append((bitmap, int(st.meta[0]), int(st.meta[1])))
    assert torch.equal(got[0][0], got[1][0])
    assert 0 < int(torch.count_nonzero(got[0][0])) and got[0][2] == got[1][2]
    # a value next to the filter's 1e-8 may fall on either side of it: sums of at most n terms in varying order
    assert abs(got[0][1] - got[1][1]) <= 2


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("rows,tile_rows_max,zipf", [(300, 64, 1.3), (2000, 512, 1.1), (5003, 1000, 1.1), (9001, 49152, 1.3), (60000, 49152, 1.1)])
def test_frequent_columns_from_row_tiles_match_the_per_column_form(binary, rows, tile_rows_max, zipf, monkeypatch):
    """Columns of one item and of many (a column in every row), tiles with ragged ends and lists that end inside a quad;
    same keys, sums equal up to the order of the adds, the same bits on every repetition."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR, GlmState
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", tile_rows_max)
    monkeypatch.setattr(T, "HOT_MIN_ENTRIES", 1)
    dev = torch.device("cuda")
    loss = L2LogLoss(1e-3)
    dim, rng = 30000, np.random.default_rng(rows)
    per = [np.unique(np.minimum(rng.zipf(zipf, rng.integers(1, 40)) - 1, dim - 1)) for _ in range(rows + 500)]
    per = [np.unique(np.concatenate([[3], p])) for p in per]      # column 3 is in every row
    rowptr = np.concatenate([[0], np.cumsum([len(p) for p in per])])
    cols = np.concatenate(per).astype(np.int32)
    vals = None if binary else torch.from_numpy(rng.normal(size=len(cols)).astype(np.float32))
    m = CSRMatrix(torch.from_numpy(rowptr), torch.from_numpy(cols), vals, torch.from_numpy(np.where(rng.random(rows + 500) < 0.5, 1.0, -1.0).astype(np.float32)), dim)
    csr = DeviceCSR(m, dev)
    w = (torch.randn(dim) * 0.3).float().to(dev)
    st = GlmState.create(dim, dim, dev)
    lo, hi = 250, 250 + rows
    plain, hot = T.build_batch_index(csr, lo, hi), T.build_batch_index(csr, lo, hi, hot=True)
    assert hot.hot is not None and (hot.hot.args.wide >= 1 or tile_rows_max <= T.HOT_SEGMENT) and torch.equal(plain.ucols, hot.ucols)
    assert hot.n_short + hot.n_medium + hot.hot.args.columns == hot.n_cols
    coef = torch.zeros((rows + 3) // 4 * 4, device=dev)
    outs = []
    for bi in (plain, hot, hot):
        out = torch.full((dim,), 7.0, device=dev)
        st.partials.zero_()
        T.glm_grad_transposed(csr, bi, w, coef, out, st.partials, st.status, loss.loss_id, loss.lam)
        assert int(st.status.item()) == 0
        outs.append(out[:bi.n_cols].clone())
    assert torch.equal(outs[1], outs[2])
    # the coefficients are at most 1 / rows in size: a sum of n products in any order is within n * 2^-24 * sum |terms|
    r_of = torch.repeat_interleave(torch.arange(rows, device=dev), csr.rowptr[lo + 1:hi + 1] - csr.rowptr[lo:hi])
    e0, e1 = int(csr.rowptr[lo]), int(csr.rowptr[hi])
    x = torch.ones(e1 - e0, device=dev, dtype=torch.float64) if binary else csr.values[e0:e1].double()
    exact = torch.zeros(dim, device=dev, dtype=torch.float64).index_add_(0, csr.cols[e0:e1].long(), coef[r_of].double() * x)
    size = torch.zeros(dim, device=dev, dtype=torch.float64).index_add_(0, csr.cols[e0:e1].long(), (coef[r_of].double() * x).abs())
    uc = hot.ucols.long()
    want = exact[uc] + loss.lam * w[uc].double()
    bound = 2 ** -20 * (size[uc] + loss.lam * w[uc].double().abs()) + 1e-12
    assert bool(((outs[1].double() - want).abs() <= bound).all())


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("rows,tile_rows_max,nnz,dim", [(200_000, 2000, 20, 10_000),   # two to four entries a list: mostly padding and bounds
                                                      (200_000, 49152, 20, 300), (100_000, 49152, 30, 100_000)])
def test_frequent_column_lists_keep_to_their_budget(rows, tile_rows_max, nnz, dim, binary, monkeypatch):
    """A budget below what building them takes is refused before it is exceeded, whatever the lists look like; twice as
    much is enough."""
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", tile_rows_max)
    monkeypatch.setattr(T, "HOT_MIN_ENTRIES", 1)
    g = torch.Generator(device="cuda").manual_seed(rows)
    cols = (dim * torch.rand(rows * nnz, generator=g, device="cuda") ** 1.5).long().clamp_(max=dim - 1)
    order = torch.argsort(cols, stable=True)
    rowidx = (order // nnz).to(torch.int32)      # (a column may hold a row twice: the lists do not mind)
    ucols, cnt = torch.unique_consecutive(cols[order], return_counts=True)
    colptr = torch.zeros(ucols.numel() + 1, dtype=torch.int32, device="cuda")
    colptr[1:] = torch.cumsum(cnt, 0)
    svals = None if binary else torch.rand(rows * nnz, generator=g, device="cuda")
    args = (ucols, colptr, rowidx, svals, cnt, rows)

    def peak(budget):
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        h, _ = T._hot_columns(*args, budget)
        scratch = 4 * h.partial_floats if h is not None else 0
        return h, max(torch.cuda.max_memory_allocated() - before, torch.cuda.memory_allocated() - before + scratch)

    h, need = peak(None)
    assert h is not None and need >= 4 * cols.numel() / 2
    del h
    for budget in (need - (64 << 10), need // 2, need // 8, 0):      # (an allocation is rounded up to 512 bytes)
        h, took = peak(budget)
        assert h is None and took <= budget + cnt.numel() * 24 + (64 << 10)   # (which columns are frequent is looked at in any case)
    h, _ = peak(2 * need)
    assert h is not None


@pytest.mark.parametrize("count", [3, 20])       # a lane's column, eight lanes' column
def test_a_column_that_ends_at_the_last_entry_there_can_be(count):
    """Entries are counted in 32 bits: a lane's steps past the end of a column that ends just below 2^31 do not come back
    as entries."""
    import ctypes
    from sketchml_b200.ops import lib as L
    last, rows = 2 ** 31 - 1, 64
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    rowidx = torch.zeros(last, dtype=torch.int32, device="cuda")
    rowidx[last - count:] = torch.arange(count, device="cuda", dtype=torch.int32)
    coef, w, out = torch.rand(rows, device="cuda"), torch.zeros(2, device="cuda"), torch.full((2,), 7.0, device="cuda")
    bins, colptr, ucols = ints(0), ints(last - count, last), ints(0, 1)
    ptr, info, loc, partial = ints(0, 0), ints(1, 0, 1, 1), torch.full((4,), rows, dtype=torch.int16, device="cuda"), torch.zeros(1, device="cuda")
    h = L.HotColumnsArgs(rows=rows, row_tiles=1, tile_rows=rows, columns=1, items=1, wide=0, info=L.ptr(info), ptr=L.ptr(ptr), loc=L.ptr(loc),
                         partial=L.ptr(partial))
    L.check(L.lib().skml_hot_colsum(ctypes.byref(h), L.ptr(bins), int(count <= 4), int(count > 4), L.ptr(colptr), L.ptr(rowidx), None, L.ptr(ucols),
                                    L.ptr(coef), L.ptr(w), 0.0, L.ptr(out), None, None, L.stream()), "skml_hot_colsum")
    want = float(coef[:count].double().sum())
    assert abs(float(out[0]) - want) <= 1e-6 * want and float(out[1]) == 0.0


def test_frequent_column_sums_on_two_streams_at_once(monkeypatch):
    """Two gradients from one batch's index at the same time have scratch of their own; the index keeps none."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.models.loss import L2LogLoss
    from sketchml_b200.ops import DeviceCSR
    from sketchml_b200.ops import transposed as T
    monkeypatch.setattr(T, "TILE_ROWS_MAX", 4096)
    monkeypatch.setattr(T, "HOT_MIN_ENTRIES", 1)
    rows, dim, nnz, dev = 120_000, 20_000, 20, torch.device("cuda")
    g = torch.Generator().manual_seed(4)
    cols = (dim * torch.rand((rows, nnz), generator=g) ** 3).int().clamp_(max=dim - 1).sort(1).values.flatten()
    csr = DeviceCSR(CSRMatrix(torch.arange(rows + 1) * nnz, cols, None, torch.sign(torch.rand(rows, generator=g) - 0.5), dim), dev)
    bi, loss = T.build_batch_index(csr, 0, rows, hot=True), L2LogLoss(1e-3)
    assert bi.hot is not None
    ws = [(torch.randn(dim, generator=g) * 0.3).to(dev) for _ in range(2)]
    state = [(torch.zeros(rows, device=dev), torch.zeros(dim, device=dev), torch.zeros(4, dtype=torch.float64, device=dev),
              torch.zeros(1, dtype=torch.int32, device=dev)) for _ in range(2)]

    def grad(i):
        T.glm_grad_transposed(csr, bi, ws[i], *state[i], loss.loss_id, loss.lam)

    want = []
    for i in range(2):
        grad(i)
        torch.cuda.synchronize()
        want.append(state[i][1].clone())
    assert not bi.hot.args.partial
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        for i in range(2):
            state[i][1].zero_()
        torch.cuda.synchronize()
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                grad(i)
        torch.cuda.synchronize()
        assert all(torch.equal(state[i][1], want[i]) for i in range(2))
