"""End-to-end training on one GPU: fused sketch path vs the uncompressed baselines and the
host engine."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _conf(**kw):
    from sketchml_b200.config import MLConf
    base = dict(algo="lr", format="synthetic", feature_num=50000, syn_rows=40000, syn_nnz_per_row=20, epoch_num=3,
                learn_rate=0.5, l2_reg=1e-4, valid_ratio=0.1, batch_sample_ratio=0.1, quant_bin_num=128,
                sketch_row_num=3, sketch_col_ratio=0.2, device="cuda", seed=1)
    base.update(kw)
    return MLConf(**base)


def _train(conf, matrix=None):
    from sketchml_b200.trainer import Trainer
    t = Trainer(conf)
    t.load_data(matrix)
    h = t.train()
    w = t.model.weights.detach().cpu().clone()
    t.close()
    return h, w, t


@pytest.mark.parametrize("algo,opt", [("lr", "sgd"), ("svm", "sgd"), ("lr", "adam"), ("linreg", "sgd")])
def test_sketch_training_tracks_uncompressed(algo, opt):
    kw = dict(algo=algo, optimizer=opt)
    if opt == "adam":
        kw["learn_rate"] = 0.01
    if algo == "linreg":
        kw.update(learn_rate=0.05, syn_values="normal", syn_wstar_density=1.0, syn_noise=0.1, feature_num=2000,
                  syn_nnz_per_row=50, syn_zipf_s=0.0)
    h_s, w_s, t_s = _train(_conf(compressor="Sketch", **kw))
    h_n, w_n, _ = _train(_conf(compressor="None", **kw))
    assert all(np.isfinite(h_s["train_loss"])) and all(np.isfinite(h_n["train_loss"]))
    assert h_n["train_loss"][-1] < h_n["train_loss"][0]
    assert h_s["train_loss"][-1] < h_s["train_loss"][0]
    # the sketch underestimates magnitudes, so it trails the exact gradient a little
    gap = abs(h_s["valid_loss"][-1] - h_n["valid_loss"][-1]) / abs(h_n["valid_loss"][-1])
    print("GAP", algo, opt, gap, h_s["valid_loss"], h_n["valid_loss"])
    assert gap < 0.3, (h_s, h_n)


def test_wire_codecs_are_lossless_and_shrink_the_payload():
    """The key encoder (delta_binary / the reference's delta_adaptive) and the table coder (8/16-bit
    cells / Huffman, the reference's wire form) only change the bytes: the trained weights are
    bit-identical for the four combinations, and every reference codec makes the payload smaller."""
    sizes, weights = {}, {}
    for enc in ("delta_binary", "delta_adaptive"):
        for cb in (-1, 0):
            from sketchml_b200.trainer import Trainer
            t = Trainer(_conf(compressor="Sketch", key_encoder=enc, cell_bits=cb, feature_num=400000, syn_rows=60000,
                              syn_nnz_per_row=30, epoch_num=1, quant_bin_num=256, valid_ratio=0.0))
            t.load_data()
            t.train()
            nnz, nbytes = t.engine.payload_stats(t.step - 1)
            sizes[(enc, cb)] = nbytes / nnz
            weights[(enc, cb)] = t.model.weights.detach().cpu().clone()
            t.close()
    print("payload bytes per non-zero", sizes)
    ref = weights[("delta_binary", -1)]
    differ = [k for k, w in weights.items() if not torch.equal(w, ref)]
    assert not differ, f"weights differ from the delta_binary / plain-table run for {differ}"
    assert sizes[("delta_adaptive", -1)] < sizes[("delta_binary", -1)]
    assert sizes[("delta_binary", 0)] < sizes[("delta_binary", -1)]
    assert sizes[("delta_adaptive", 0)] == min(sizes.values())


@pytest.mark.parametrize("opt", ["sgd", "adam"])
def test_running_weight_norm_matches_a_pass_over_the_model(opt):
    """The decode kernel keeps sum(w^2) current while it updates (no pass over the model per step): the
    per-epoch losses equal those of a run that recomputes the norm every step, and the running sum
    equals the model's at the end."""
    from sketchml_b200.trainer import Trainer
    kw = dict(compressor="Sketch", optimizer=opt, learn_rate=0.5 if opt == "sgd" else 0.01, l2_reg=1e-2, valid_ratio=0.0,
              epoch_num=2)
    res = {}
    for track in (True, False):
        t = Trainer(_conf(extras={"track_norm": track}, **kw))
        t.load_data()
        h = t.train()
        w = t.model.weights.detach().double()
        res[track] = (h["train_loss"], w.clone(), float(t.engine.wsq.item()))
        assert (t.engine.dec.norm_track is not None) == track
        t.close()
    assert torch.equal(res[True][1], res[False][1])
    assert np.allclose(res[True][0], res[False][0], rtol=1e-6, atol=0)
    true_sq = float((res[True][1] ** 2).sum())
    assert abs(res[True][2] - true_sq) <= 1e-5 * true_sq, (res[True][2], true_sq)


def test_gpu_uncompressed_matches_host_engine():
    from sketchml_b200.data import SyntheticSpec, generate_cpu
    spec = SyntheticSpec(6000, 8000, 15, 1.1, "binary", "logistic", 0.1, 0.0, 3)
    m, _ = generate_cpu(spec)
    kw = dict(feature_num=8000, epoch_num=2, valid_ratio=0.2, compressor="None", l2_reg=1e-3)
    h_g, w_g, _ = _train(_conf(**kw), m)
    h_c, w_c, _ = _train(_conf(device="cpu", dtype="float64", **kw), m)
    assert np.allclose(h_g["train_loss"], h_c["train_loss"], rtol=2e-4)
    assert np.allclose(h_g["valid_loss"], h_c["valid_loss"], rtol=2e-4)
    assert float((w_g.double() - w_c.double()).abs().max()) < 1e-4


def test_kv_baseline_and_checkpoint_resume(tmp_path):
    h1, w1, _ = _train(_conf(compressor="Float", epoch_num=2))
    h2, w2, _ = _train(_conf(compressor="None", epoch_num=2))
    assert float((w1 - w2).abs().max()) < 1e-5
    ck = tmp_path / "ck"
    _train(_conf(compressor="Sketch", epoch_num=1, checkpoint_dir=str(ck), checkpoint_every=1))
    h3, w3, _ = _train(_conf(compressor="Sketch", epoch_num=2, resume=str(ck / "epoch_0001.ckpt")))
    h4, w4, _ = _train(_conf(compressor="Sketch", epoch_num=2))
    assert len(h3["train_loss"]) == 1
    # float atomics make two runs differ in the last bits, which can move a value across a bucket edge
    assert float((w3 - w4).abs().mean()) < 2e-4 and float((w3 - w4).abs().max()) < 0.2


def test_pipeline_depth_one_trains_like_depth_zero():
    h0, w0, _ = _train(_conf(compressor="Sketch", epoch_num=3))
    h1, w1, _ = _train(_conf(compressor="Sketch", epoch_num=3, pipeline_depth=1))
    assert h1["train_loss"][-1] < h1["train_loss"][0]
    # a gradient that is one step stale costs a little progress, not convergence
    assert abs(h1["valid_loss"][-1] - h0["valid_loss"][-1]) / h0["valid_loss"][-1] < 0.01


@pytest.mark.parametrize("name", ["FixedPoint", "Zip"])
def test_baseline_compressors_train_on_gpu(name):
    h, w, _ = _train(_conf(compressor=name, epoch_num=2, quant_bin_num=64))
    h0, w0, _ = _train(_conf(compressor="None", epoch_num=2))
    assert h["train_loss"][-1] < h["train_loss"][0]
    assert abs(h["valid_loss"][-1] - h0["valid_loss"][-1]) / h0["valid_loss"][-1] < 0.05


def test_transposed_index_path_trains_like_scatter_path():
    kw = dict(compressor="Sketch", epoch_num=2, valid_ratio=0.0, syn_rows=30000, batch_sample_ratio=0.1)
    h_t, w_t, t_t = _train(_conf(**kw))
    assert t_t.engine.tindex is not None and len(t_t.engine.tindex) == 10
    h_s, w_s, t_s = _train(_conf(extras={"transposed_index": False}, **kw))
    assert t_s.engine.tindex is None
    # the scatter path sums with float atomics, so its gradients differ in the last bits from run
    # to run; bucket boundaries and sketch collisions amplify that to a few 1e-3 of the loss. The index path repeats
    # bit for bit. Sixty runs of the scatter form: its losses spread with a standard deviation of 0.18 % around a mean
    # 0.2 % from the index form's (largest difference 0.55 %), the weights by 6.5e-5 at most: the bounds lie more than
    # four standard deviations out.
    assert np.allclose(h_t["train_loss"], h_s["train_loss"], rtol=1e-2)
    assert float((w_t - w_s).abs().mean()) < 2e-3


def test_packed_batch_transport_matches_plain_and_trains():
    """The bit-packed host->device batch form expands to exactly the plain CSR arrays, and a
    streamed run through it equals a streamed run through the plain form."""
    from sketchml_b200.data import HostBatchFeeder, PinnedBatch, SyntheticSpec, generate_cpu
    from sketchml_b200.data.dataset import CSRMatrix
    from sketchml_b200.trainer import Trainer
    spec = SyntheticSpec(6000, 40001, 12, 1.1, "binary", "logistic", 0.1, 0.0, 5)
    m, _ = generate_cpu(spec)
    B = 1500
    parts = []
    for i in range(4):
        lo, hi = int(m.rowptr[i * B]), int(m.rowptr[(i + 1) * B])
        parts.append(CSRMatrix(m.rowptr[i * B:(i + 1) * B + 1].clone(), m.cols[lo:hi].clone(), None,
                               m.labels[i * B:(i + 1) * B].clone(), m.dim))
    plain = HostBatchFeeder([PinnedBatch(p) for p in parts], "cuda")
    packed = HostBatchFeeder([PinnedBatch(p, packed=True, transport="bits") for p in parts], "cuda")
    varb = HostBatchFeeder([PinnedBatch(p, packed=True, transport="varbytes") for p in parts], "cuda")
    varn = HostBatchFeeder([PinnedBatch(p, packed=True, transport="varnibbles") for p in parts], "cuda")
    auto = PinnedBatch(parts[0], packed=True)
    assert packed.batches[0].bits == 16 and packed.batches[0].labels8 and not packed.batches[0].varbytes
    assert packed.batches[0].h2d_bytes() < 0.62 * plain.batches[0].h2d_bytes()
    assert auto.h2d_bytes() == min(packed.batches[0].h2d_bytes(), varb.batches[0].h2d_bytes(), varn.batches[0].h2d_bytes())
    for i in range(4):
        plain.prefetch(i)
        a, rows = plain.get(i)
        for other in (packed, varb, varn):
            other.prefetch(i)
            b, rows_b = other.get(i)
            torch.cuda.synchronize()
            assert rows == rows_b == B
            n = parts[i].nnz
            assert torch.equal(a.rowptr[:B + 1], b.rowptr[:B + 1])
            assert torch.equal(a.cols[:n], b.cols[:n])
            assert torch.equal(a.labels[:B], b.labels[:B])
            other.release(i)
        plain.release(i)
    ws = []
    for feeder in (plain, packed, varb):
        t = Trainer(_conf(feature_num=m.dim, compressor="None", valid_ratio=0.0, batch_sample_ratio=0.25))
        t.load_data(m)
        t.train_streamed(feeder, 4)
        torch.cuda.synchronize()
        ws.append(t.model.weights.detach().cpu().clone())
        t.close()
    assert float((ws[0] - ws[1]).abs().max()) < 1e-6 and float((ws[0] - ws[2]).abs().max()) < 1e-6


@pytest.mark.parametrize("transposed", [True, False])
def test_shadow_mode_recomputes_every_payload_on_the_cpu(transposed):
    """Debug mode: each step's payload equals the oracle's for the same keys, values and splits."""
    kw = dict(compressor="Sketch", epoch_num=1, valid_ratio=0.0, syn_rows=20000, batch_sample_ratio=0.1,
              extras={"shadow_every": 1, "transposed_index": transposed})
    h, w, t = _train(_conf(**kw))
    assert t.engine.shadow_checks == 10
    assert (t.engine.tindex is not None) == transposed


def test_shadow_compare_reports_a_wrong_payload():
    from sketchml_b200.ops import GpuCompressor
    from sketchml_b200.utils.shadow import ShadowMismatch, check_payload, compare_payload
    rng = np.random.default_rng(0)
    dim, n = 100000, 6000
    keys = np.sort(rng.choice(dim, n, replace=False)).astype(np.int32)
    vals = rng.laplace(0, 1e-3, n).astype(np.float32)
    comp = GpuCompressor(dim, n, 128, 8, 3, 0.2, seed=9)
    buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=4, rank=1, world=2)
    payload = comp.payload_bytes(buf)
    splits = comp.last_splits()
    assert compare_payload(payload, keys, vals, dim, splits, 8, 3, 0.2, 9) == []
    wrong = vals.copy()
    wrong[::7] *= -3.0
    with pytest.raises(ShadowMismatch):
        check_payload(payload, keys, wrong, dim, splits, 8, 3, 0.2, 9)


def test_local_id_batches_train_like_plain_streamed_batches():
    """Streamed batches whose columns were replaced by batch-local ids on the host (the device
    scatters into a compact accumulator, no bitmap compaction) give the plain streamed result, and
    their payloads pass the shadow check."""
    from sketchml_b200.data import HostBatchFeeder, PinnedBatch, SyntheticSpec, generate_cpu
    from sketchml_b200.data.dataset import CSRMatrix
    from sketchml_b200.trainer import Trainer
    spec = SyntheticSpec(8000, 60001, 15, 1.1, "binary", "logistic", 0.1, 0.0, 6)
    m, _ = generate_cpu(spec)
    B = 2000
    parts = []
    for i in range(4):
        lo, hi = int(m.rowptr[i * B]), int(m.rowptr[(i + 1) * B])
        parts.append(CSRMatrix(m.rowptr[i * B:(i + 1) * B + 1].clone(), m.cols[lo:hi].clone(), None,
                               m.labels[i * B:(i + 1) * B].clone(), m.dim))
    local = [PinnedBatch(p, local_ids=True) for p in parts]
    assert local[0].n_cols == len(np.unique(parts[0].cols.numpy())) and local[0].packed
    ws, losses = [], []
    for batches in ([PinnedBatch(p, packed=True) for p in parts], local):
        feeder = HostBatchFeeder(batches, "cuda")
        t = Trainer(_conf(feature_num=m.dim, compressor="Sketch", valid_ratio=0.0, batch_sample_ratio=0.25,
                          extras={"shadow_every": 1}))
        t.load_data(m)
        lh = t.train_streamed(feeder, 8)
        torch.cuda.synchronize()
        t.engine.check()
        assert t.engine.shadow_checks == 8
        ws.append(t.model.weights.detach().cpu().clone())
        losses.append((lh[:, 1] / lh[:, 0]).numpy())
        t.close()
    # float atomics order differs between the two scatters: bucket edges may move a value, as between two runs
    assert np.allclose(losses[0], losses[1], rtol=2e-3)
    assert float((ws[0] - ws[1]).abs().mean()) < 2e-3


@pytest.mark.parametrize("opt", ["sgd", "adam"])
@pytest.mark.parametrize("name", ["Float", "FixedPoint", "Zip"])
def test_baseline_step_behind_one_call_equals_its_separate_calls(name, opt):
    """Batches of 400 rows keep every column below the length that is summed with atomics, so both forms of the step
    run the same sums in the same order: the same weights, bit for bit."""
    kw = dict(compressor=name, optimizer=opt, epoch_num=2, valid_ratio=0.0, syn_rows=2000, batch_sample_ratio=0.2, quant_bin_num=64,
              learn_rate=0.5 if opt == "sgd" else 0.01)
    h1, w1, _ = _train(_conf(**kw))
    h2, w2, _ = _train(_conf(extras={"single_call_step": False}, **kw))
    assert torch.equal(w1, w2)
    assert np.allclose(h1["train_loss"], h2["train_loss"], rtol=1e-12)


@pytest.mark.parametrize("single_call", [True, False])
@pytest.mark.parametrize("opt", ["sgd", "adam"])
@pytest.mark.parametrize("rows", [1000, 60000])
def test_zip_step_after_a_reported_error_changes_nothing_and_is_raised(rows, opt, single_call):
    """A split search that gives up at a grid barrier leaves the tables of an earlier step. Its status word (set here on
    the host, as such a search would) keeps codes, values, weights and moments as they are and reaches the engine's
    check; search by one block and by several."""
    from sketchml_b200.parallel.failure import STATUS_TIMEOUT_BARRIER, StepTimeout
    from sketchml_b200.trainer import Trainer
    t = Trainer(_conf(compressor="Zip", optimizer=opt, valid_ratio=0.0, syn_rows=rows, feature_num=2000000, batch_sample_ratio=0.5,
                      quant_bin_num=64, learn_rate=0.5 if opt == "sgd" else 0.01, extras={"single_call_step": single_call}))
    t.load_data()
    t.train_one_iteration(0, 0)
    eng = t.engine
    state = [t.model.weights] + ([t.model.optimizer.m, t.model.optimizer.v] if opt == "adam" else []) + [eng.zip_codec.codes]
    before = [x.clone() for x in state]
    eng.st.status.fill_(STATUS_TIMEOUT_BARRIER | 0x6200)
    t.train_one_iteration(0, 1)
    assert all(torch.equal(a, b) for a, b in zip(before[:-1], state[:-1]))
    assert torch.equal(before[-1], state[-1])
    with pytest.raises(StepTimeout):
        eng.check()
    t.train_one_iteration(0, 2)    # the word is clear again: the next step counts
    eng.check()
    assert not torch.equal(before[0], state[0])
    t.close()


def test_a_step_of_over_a_million_columns():
    """The number of keys comes from the column index and the device: the sketch is inserted in shared memory, which has a
    stage of its own between scatter and key code; the weights are those of the staged launches, which insert with atomics."""
    from sketchml_b200.trainer import Trainer
    ws = []
    for fused in (True, False):
        t = Trainer(_conf(feature_num=3_000_000, syn_rows=120_000, syn_nnz_per_row=30, syn_zipf_s=0.0, valid_ratio=0.0, batch_sample_ratio=0.5,
                          quant_bin_num=256, extras={"fused": fused}))
        t.load_data()
        assert all(bi.n_cols > 1_000_000 for bi in t.engine.tindex)
        for i in range(2):
            t.train_one_iteration(0, i)
        if fused:
            st = t.engine.stage_times_us()
            total = sum(st["compress"])
            assert 0 < st["sketch_insert"] < st["compress"][3] < total    # the scatter's stage holds it
            assert st["sketch_insert"] > st["compress"][4] / 8            # (it was counted as key code)
        ws.append(t.model.weights.detach().cpu().clone())
        t.close()
    assert torch.count_nonzero(ws[0]) > 1_000_000 and torch.equal(ws[0], ws[1])


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("compressor", ["Float", "Sketch"])
def test_steps_with_lists_of_frequent_columns_train_like_steps_without(compressor, binary, monkeypatch):
    """Three batches of a data set, of which two have lists of frequent columns, of different sizes, and share their
    scratch: losses (settled by the kernel that adds the partial sums) and weights over two epochs."""
    from sketchml_b200.data import CSRMatrix
    from sketchml_b200.ops import transposed as T
    from sketchml_b200.trainer import Trainer
    B, nnz, dim = 20000, 20, 1_000_000
    g = torch.Generator().manual_seed(7)
    u = torch.rand((3 * B, nnz), generator=g, dtype=torch.float64)
    u[:B] **= 12                       # batch 0 most frequent, batch 1 every column alike, batch 2 in between
    u[2 * B:] **= 6
    cols = (dim * u).int().clamp_(max=dim - 1).sort(1).values
    keep = torch.ones_like(cols, dtype=torch.bool)
    keep[:, 1:] = cols[:, 1:] != cols[:, :-1]
    rowptr = torch.zeros(3 * B + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(keep.sum(1), 0)
    vals = None if binary else torch.randn(int(rowptr[-1]), generator=g)
    m = CSRMatrix(rowptr, cols[keep], vals, torch.sign(torch.rand(3 * B, generator=g) - 0.4), dim)
    monkeypatch.setattr(T, "TILE_ROWS_MAX", 6000)
    got = []
    for least in (50_000, 10 ** 12):
        monkeypatch.setattr(T, "HOT_MIN_ENTRIES", least)
        t = Trainer(_conf(compressor=compressor, feature_num=dim, valid_ratio=0.0, batch_sample_ratio=1 / 3, quant_bin_num=256))
        t.load_data(m)
        hot = [bi.hot for bi in t.engine.tindex]
        assert [h is not None for h in hot] == [least == 50_000, False, least == 50_000]
        if least == 50_000:
            assert hot[0].args.partial == hot[2].args.partial and hot[0].partial_floats != hot[2].partial_floats
        # weights in the middle of a training: no two coefficients alike, so that no crowd of equal sums lies on a bucket's border
        t.model.weights.normal_(0.0, 0.01, generator=torch.Generator(device="cuda").manual_seed(3))
        t.engine.after_resume()
        start = t.model.weights.detach().cpu().clone()
        losses = []
        for epoch in range(2):
            for i in range(3):
                t.train_one_iteration(epoch, i)
            losses.append(t.engine.loss_ring.cpu().clone())
        got.append((torch.stack(losses), t.model.weights.detach().cpu().clone()))
        t.close()
    (l0, w0), (l1, w1) = got
    assert float(l0[..., 1].abs().min()) > 0
    if compressor == "Float":     # sums of the same fp32 terms in another order
        assert torch.allclose(l0, l1, rtol=1e-6) and torch.allclose(w0, w1, rtol=1e-4, atol=1e-8)
    else:   # a sum within rounding of a bucket's border (some 1e-6 of them) may change its bucket, and the cells it is least in
        assert torch.allclose(l0[0, 0], l1[0, 0], rtol=1e-9) and torch.allclose(l0, l1, rtol=1e-5)
        assert float((w0 - w1).norm()) <= 1e-2 * float((w1 - start).norm())
