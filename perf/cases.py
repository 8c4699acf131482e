"""Workloads of the framework's public entry points, with the work each one cannot do without.

`listed()` holds the workloads by name, `draw()` makes more of the same ranges, `prepare()` builds what a
program has in hand before the call, `run()` is one pass of the call. Kinds of workload:

* ``epoch``   a whole training epoch and its validation through `Trainer.train_one_epoch` / `Trainer.validate`
* ``step``    one minibatch step through `Trainer.train_one_iteration` on a resident shard
* ``stream``  four steps through `Trainer.train_streamed`, every batch copied from pinned host memory
* ``codec``   one gradient through the stand-alone device codec and back (`GpuCompressor` / `GpuDecoder`)
* ``encode``  one gradient through `GpuCompressor.compress_local` alone (what a sender does)
* ``decode``  the payloads of several ranks through `GpuDecoder.decode_update` (what every receiver does)
* ``keys``    a sorted key list through the stand-alone delta-adaptive codec and back (`ops.keys`)
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

STREAM_STEPS = 4
RAGGED_SHARE = 0.7


# --------------------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------------------
def _train(kind, algo, features, rows, batch, nnz, **more):
    c = dict(kind=kind, algo=algo, features=int(features), rows=int(rows), batch=float(batch), nnz=int(nnz), zipf=1.1,
             values="binary", valid=0.0, optimizer="sgd", compressor="Sketch", bins=256, sketch_rows=3, sketch_cols=0.2,
             key_encoder="delta_binary", cell_bits=-1, ragged=False)
    c.update(more)
    return c


def listed():
    return [
        # A first run on a small data set with the option defaults of the original (Adam, a quarter of the rows held
        # out, 2 x 0.3 sketches): 10 batches of about 7,500 rows and the validation; bound by launches and host work.
        dict(_train("epoch", "lr", 100_000, 100_000, 0.1, 20, valid=0.25, optimizer="adam", sketch_rows=2, sketch_cols=0.3),
             name="epoch_lr_100k_adam"),
        # One GPU's share of the headline logistic regression on eight GPUs (62,500 of 500,000 rows per step).
        dict(_train("step", "lr", 50_000_000, 125_000, 0.5, 30), name="step_lr_50m_shard"),
        # The headline logistic regression on one GPU: 500,000 rows of 30 binary features per step, 50M features.
        dict(_train("step", "lr", 50_000_000, 1_000_000, 0.5, 30), name="step_lr_50m"),
        # The linear SVM configuration: 1M rows of 30 real values per step, 100M features, 64 buckets.
        dict(_train("step", "svm", 100_000_000, 2_000_000, 0.5, 30, zipf=1.2, values="uniform_l2", bins=64), name="step_svm_100m"),
        # The least-squares configuration: 500,000 rows of 200 values, 1M features: nearly dense gradients, which
        # take the dense kind of payload.
        dict(_train("step", "linreg", 1_000_000, 500_000, 1.0, 200, zipf=0.0, values="normal"), name="step_linreg_1m_dense"),
        # The original's wire options (adaptive key code, Huffman-coded tables) with Adam, held-out rows and rows of
        # different lengths.
        dict(_train("step", "lr", 4_000_000, 200_000, 0.25, 30, valid=0.25, optimizer="adam", sketch_rows=2, sketch_cols=0.3,
                    key_encoder="delta_adaptive", cell_bits=0, ragged=True), name="step_lr_4m_adam_wire"),
        # Data that does not stay resident: plain CSR batches of 100,000 rows from pinned host memory.
        dict(_train("stream", "lr", 10_000_000, 100_000, 1.0, 30, ragged=True), name="stream_lr_10m"),
        # The ZipML comparison compressor in a training step (users compare compressors on one data set).
        dict(_train("step", "lr", 4_000_000, 80_000, 0.5, 30, compressor="Zip"), name="step_lr_4m_zip"),
        # The library demo: a sparse vector of 100,000 dimensions with one non-zero in ten, there and back.
        dict(kind="codec", dim=100_000, n=10_000, bins=256, sketch_rows=2, sketch_cols=0.3, dense=False, name="codec_demo_10k"),
        # The sender's side of the compression microbenchmark at its largest: 10M non-zeros of 100M.
        dict(kind="encode", dim=100_000_000, n=10_000_000, bins=256, sketch_rows=3, sketch_cols=0.2, name="encode_10m_of_100m"),
        # The receiver's side of the headline configuration on eight GPUs: eight payloads of one 62,500-row batch each.
        dict(kind="decode", dim=50_000_000, ranks=8, rows=62_500, nnz=30, zipf=1.1, bins=256, sketch_rows=3, sketch_cols=0.2,
             optimizer="sgd", name="decode_8_ranks_50m"),
        # A library call on a key list of the microbenchmark's smaller size.
        dict(kind="keys", dim=100_000_000, n=1_000_000, name="keys_1m_of_100m"),
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["epoch", "step", "step", "step", "stream", "baseline", "codec", "encode", "decode", "keys"])
    if kind == "epoch":
        return _train("epoch", rng.choice(["lr", "svm", "linreg"]), _log_int(rng, 20_000, 1_000_000), _log_int(rng, 10_000, 120_000),
                      0.1, rng.randint(5, 40), valid=0.25, optimizer=rng.choice(["adam", "sgd"]), sketch_rows=2, sketch_cols=0.3,
                      values=rng.choice(["binary", "uniform_l2"]), ragged=rng.random() < 0.5)
    if kind == "step":
        algo = rng.choice(["lr", "lr", "svm", "linreg"])
        if algo == "linreg":
            batch_rows, nnz = _log_int(rng, 20_000, 400_000), rng.randint(60, 200)
            dim = _log_int(rng, 200_000, 1_000_000)
            return _train("step", algo, dim, batch_rows, 1.0, nnz, zipf=0.0, values="normal")
        batch_rows, nnz = _log_int(rng, 3_000, 500_000), rng.randint(8, 40)
        held = rng.random() < 0.4          # held-out rows: the shard is no whole number of batches
        more = dict(valid=0.25) if held else {}
        if rng.random() < 0.3:
            more.update(optimizer="adam", sketch_rows=2, sketch_cols=0.3)
        if rng.random() < 0.25:
            more.update(key_encoder="delta_adaptive", cell_bits=0)
        return _train("step", algo, _log_int(rng, 1_000_000, 80_000_000), 2 * batch_rows, 0.5, nnz,
                      zipf=rng.choice([1.1, 1.2]), values="binary" if algo == "lr" else "uniform_l2",
                      bins=rng.choice([64, 128, 256]), ragged=rng.random() < 0.5, **more)
    if kind == "baseline":
        return _train("step", "lr", _log_int(rng, 400_000, 4_000_000), 2 * _log_int(rng, 4_000, 40_000), 0.5, rng.randint(10, 30),
                      compressor=rng.choice(["Zip", "FixedPoint"]))
    if kind == "stream":
        return _train("stream", "lr", _log_int(rng, 500_000, 10_000_000), _log_int(rng, 5_000, 100_000), 1.0, rng.randint(10, 30),
                      ragged=rng.random() < 0.5)
    if kind == "codec":
        dim = _log_int(rng, 20_000, 2_000_000)
        dense = rng.random() < 0.4
        return dict(kind="codec", dim=dim, n=dim if dense else max(1_000, int(dim * rng.uniform(0.02, 0.3))),
                    bins=rng.choice([64, 128, 256]), sketch_rows=2, sketch_cols=0.3, dense=dense)
    if kind == "encode":
        n = _log_int(rng, 100_000, 10_000_000)
        return dict(kind="encode", dim=int(n * rng.choice([10, 100])) if n <= 1_000_000 else 10 * n, n=n,
                    bins=rng.choice([64, 128, 256]), sketch_rows=3, sketch_cols=0.2)
    if kind == "decode":
        return dict(kind="decode", dim=_log_int(rng, 2_000_000, 50_000_000), ranks=rng.choice([2, 4, 8]), rows=_log_int(rng, 2_000, 62_500),
                    nnz=rng.randint(10, 30), zipf=1.1, bins=rng.choice([64, 256]), sketch_rows=3, sketch_cols=0.2,
                    optimizer=rng.choice(["sgd", "adam"]))
    n = _log_int(rng, 10_000, 1_000_000)
    return dict(kind="keys", dim=n * rng.randint(3, 100), n=n)


# --------------------------------------------------------------------------------------------------
# what a program has in hand before the call
# --------------------------------------------------------------------------------------------------
def _gradient(dim, n, gen):
    """Sorted distinct uniform keys and Laplace(0, 1e-3) values."""
    k = torch.randint(0, dim, (int(n * 1.25) + 64,), generator=gen, device="cuda", dtype=torch.int32)
    k = torch.unique(k)
    while k.numel() < n:
        more = torch.randint(0, dim, (n,), generator=gen, device="cuda", dtype=torch.int32)
        k = torch.unique(torch.cat([k, more]))
    if k.numel() > n:
        k = k[torch.randperm(k.numel(), generator=gen, device="cuda")[:n].sort().values]
    return k.contiguous(), _laplace(n, gen)


def _laplace(n, gen):
    u = (torch.rand(n, generator=gen, device="cuda") - 0.5).clamp(-0.4999999, 0.4999999)
    v = -1e-3 * torch.sign(u) * torch.log1p(-2 * u.abs())
    return torch.where(v.abs() < 1e-8, torch.full_like(v, 1e-6), v).contiguous()


def _rows(case, rows, seed):
    """The case's rows on the device; ``ragged``: three entries in ten are left out, so that row lengths differ."""
    from sketchml_b200.data import CSRMatrix, SyntheticSpec
    from sketchml_b200.ops import generate_gpu
    task = {"lr": "logistic", "svm": "svm", "linreg": "regression"}[case["algo"]]
    k = case["nnz"]
    spec = SyntheticSpec(rows, case["features"], k, case["zipf"], case["values"], task, 0.01, 0.0, seed)
    m = generate_gpu(spec, 0, rows, torch.device("cuda"))[0].to_matrix()
    if not case["ragged"]:
        return m
    keep = torch.rand((rows, k), generator=torch.Generator(device="cuda").manual_seed(seed + 2), device="cuda") < RAGGED_SHARE
    keep[:, 0] = True
    rowptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(keep.sum(1), 0, out=rowptr[1:])
    keep = keep.reshape(-1)
    return CSRMatrix(rowptr, m.cols[keep], None if m.values is None else m.values[keep], m.labels, m.dim)


def _trainer(case, seed, matrix=None):
    from sketchml_b200.config import MLConf
    from sketchml_b200.trainer import Trainer
    if matrix is None and case["ragged"]:
        matrix = _rows(case, case["rows"], seed)
    extras = {"transposed_index": False} if case["kind"] == "stream" else {}
    conf = MLConf(algo=case["algo"], format="synthetic", feature_num=case["features"], valid_ratio=case["valid"], epoch_num=1,
                  batch_sample_ratio=case["batch"], learn_rate=0.01 if case["optimizer"] == "adam" else 0.05, learn_decay=0.9,
                  l2_reg=1e-5 if case["algo"] == "svm" else 1e-4, compressor=case["compressor"], quant_bin_num=case["bins"],
                  sketch_group_num=8, sketch_row_num=case["sketch_rows"], sketch_col_ratio=case["sketch_cols"],
                  optimizer=case["optimizer"], key_encoder=case["key_encoder"], cell_bits=case["cell_bits"], device="cuda",
                  seed=seed, syn_rows=case["rows"], syn_nnz_per_row=case["nnz"], syn_zipf_s=case["zipf"], syn_values=case["values"],
                  syn_wstar_density=1.0 if case["algo"] == "linreg" else 0.01, syn_noise=0.0 if case["algo"] == "lr" else 0.1,
                  extras=extras)
    t = Trainer(conf)
    t.load_data(matrix)
    if getattr(t.engine, "xchg", None) is not None:
        weakref.finalize(t, t.engine.xchg.close)    # the receive region goes back with the trainer
    # a model in the middle of its training: no weight is zero, so no two coefficients of a batch are alike
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    t.model.weights.normal_(0.0, 0.01, generator=g)
    if case["optimizer"] == "adam":
        opt = t.model.optimizer
        opt.m.copy_(torch.randn(case["features"], generator=g, device="cuda") * 1e-4)
        opt.v.copy_((torch.rand(case["features"], generator=g, device="cuda") + 0.5) * 1e-8)
    t.engine.after_resume()
    return t


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("epoch", "step"):
        return dict(kind=kind, adam=case["optimizer"] == "adam", trainer=_trainer(case, seed))
    if kind == "stream":
        from sketchml_b200.data import HostBatchFeeder, PinnedBatch
        B = case["rows"]
        m = _rows(case, STREAM_STEPS * B, seed)
        parts = [m.slice_rows(i * B, (i + 1) * B) for i in range(STREAM_STEPS)]
        feeder = HostBatchFeeder([PinnedBatch(p.to("cpu")) for p in parts], "cuda")
        loss = torch.zeros((STREAM_STEPS, 4), dtype=torch.float64).pin_memory()
        return dict(kind=kind, trainer=_trainer(case, seed, parts[0]), feeder=feeder, loss=loss)
    from sketchml_b200.ops.codec import GpuCompressor, GpuDecoder
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "keys":
        n = case["n"]       # the code's length depends on the keys: a program keeps it in a buffer that fits every list
        room = lambda bits: torch.zeros((bits * n + 63) // 64, dtype=torch.int64, device="cuda")
        return dict(kind=kind, keys=_gradient(case["dim"], n, gen)[0], flags=room(17), deltas=room(32))
    opts = dict(bin_num=case["bins"], group_num=8, row_num=case["sketch_rows"], col_ratio=case["sketch_cols"], seed=seed)
    if kind in ("codec", "encode"):
        dim, n = case["dim"], case["n"]
        dense = bool(case.get("dense"))
        keys, vals = (None, torch.randn(dim, generator=gen, device="cuda")) if dense else _gradient(dim, n, gen)
        s = dict(kind=kind, comp=GpuCompressor(dim, n, **opts), keys=keys, vals=vals, dense=dense)
        if kind == "codec":
            s["dec"] = GpuDecoder(dim, n, max_groups=8)
        return s
    # decode: one payload per rank from that rank's batch
    from sketchml_b200.data import SyntheticSpec
    from sketchml_b200.ops import generate_gpu
    P, dim, per, k = case["ranks"], case["dim"], case["rows"], case["nnz"]
    spec = SyntheticSpec(per * P, dim, k, case["zipf"], "binary", "logistic", 0.01, 0.0, seed)
    cols = generate_gpu(spec, 0, per * P, torch.device("cuda"))[0].cols
    keys = [torch.unique(cols[r * per * k:(r + 1) * per * k]).int() for r in range(P)]
    nmax = max(x.numel() for x in keys)
    comp = GpuCompressor(dim, nmax, **opts)
    payloads = [comp.compress_local(x, _laplace(x.numel(), gen), rank=r, world=P) for r, x in enumerate(keys)]
    s = dict(kind=kind, dec=GpuDecoder(dim, nmax * P, max_groups=8), payloads=payloads, capacity=comp.capacity,
             w=torch.randn(dim, generator=gen, device="cuda") * 0.01, m=None, v=None,
             status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    if case["optimizer"] == "adam":
        quad = torch.zeros((dim, 4), device="cuda")     # the engine's packed state: {m, v, sum, -} per coordinate
        quad[:, 0] = torch.randn(dim, generator=gen, device="cuda") * 1e-4
        quad[:, 1] = (torch.rand(dim, generator=gen, device="cuda") + 0.5) * 1e-8
        s.update(m=quad[:, 0], v=quad[:, 1])
    return s


# --------------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "step":
        t = s["trainer"]
        t.train_one_iteration(0, 0)
        out = [t.model.weights, t.engine.loss_ring]
        return out + [t.model.optimizer.m, t.model.optimizer.v] if s["adam"] else out
    if kind == "epoch":
        t = s["trainer"]
        loss = t.train_one_epoch(0, t.conf.batch_num)
        v = t.validate(0)
        out = [t.model.weights, loss, v["valid_loss"]]
        return out + [t.model.optimizer.m, t.model.optimizer.v] if s["adam"] else out
    if kind == "stream":
        t = s["trainer"]
        t.train_streamed(s["feeder"], STREAM_STEPS, loss_host=s["loss"])
        return [t.model.weights, s["loss"]]
    if kind == "encode":
        return s["comp"].compress_local(s["keys"], s["vals"])
    if kind == "codec":
        payload = s["comp"].compress_local(s["keys"], s["vals"], dense=s["dense"])
        return [payload, s["dec"].decode_sum([payload])]
    if kind == "decode":
        p = s["payloads"]
        s["dec"].decode_update([x.data_ptr() for x in p], [None] * len(p), s["capacity"], 0, s["status"], s["w"],
                               0.01 if s["m"] is not None else 0.05, s["m"], s["v"], 1.0)
        return [s["w"], s["status"]] + ([s["m"], s["v"]] if s["m"] is not None else [])
    from sketchml_b200.ops import keys as K
    e = K.encode(s["keys"])
    s["flags"][:e.flag_words.numel()].copy_(e.flag_words)
    s["deltas"][:e.delta_words.numel()].copy_(e.delta_words)
    return [e.size, e.num_intervals, e.flag_kind, e.flag_bits, e.delta_bits, s["flags"], s["deltas"], K.decode(e)]


# --------------------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------------------
def _distinct(dim, s, draws):
    """Expected number of distinct columns among ``draws`` Zipf(s) draws (uniform for s = 0)."""
    if s == 0.0:
        return dim * -math.expm1(draws * math.log1p(-1.0 / dim))
    edges = np.unique(np.concatenate([np.arange(1, min(dim, 4096) + 1), np.geomspace(1, dim + 1, 4000)]))
    a = 1.0 - s
    top = (dim + 1.0) ** a - 1.0
    mass = (edges[1:] ** a - edges[:-1] ** a) / top      # the density x^-s on [1, dim + 1)
    width = edges[1:] - edges[:-1]
    return float((width * -np.expm1(-draws * mass / width)).sum())


def _step_work(case, rows):
    """Batch rows read once, every touched weight (and moment) read and written once, the payload written and read."""
    nnz = rows * case["nnz"] * (RAGGED_SHARE if case["ragged"] else 1.0)
    u = _distinct(case["features"], case["zipf"], nnz)
    adam = case["optimizer"] == "adam"
    payload = {"Sketch": 2.0, "Zip": 6.0, "FixedPoint": 5.0}[case["compressor"]]   # bytes per non-zero
    return {"bytes": nnz * (4 if case["values"] == "binary" else 8) + 12 * rows + u * ((24 if adam else 8) + 2 * payload),
            "flops": 4.0 * nnz + 12.0 * u}


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _step_work(case, int(case["rows"] * (1 - case["valid"]) * case["batch"]))
    if kind == "epoch":
        w = _step_work(case, int(case["rows"] * (1 - case["valid"]) * case["batch"]))
        nv = case["rows"] * case["valid"] * case["nnz"]
        return {"bytes": 10 * w["bytes"] + nv * (4 if case["values"] == "binary" else 8), "flops": 10 * w["flops"] + 2 * nv}
    if kind == "stream":
        w = _step_work(case, case["rows"])
        return {"bytes": STREAM_STEPS * w["bytes"], "flops": STREAM_STEPS * w["flops"]}
    if kind == "keys":
        width = max(1.0, math.log2(case["dim"] / case["n"]) + 3.0) / 8.0     # bytes of a coded key
        return {"bytes": case["n"] * 2 * (4 + width), "flops": 4.0 * case["n"]}
    if kind == "decode":
        n = _distinct(case["dim"], case["zipf"], case["rows"] * case["nnz"])
        u = _distinct(case["dim"], case["zipf"], case["ranks"] * case["rows"] * case["nnz"])
        return {"bytes": case["ranks"] * n * 2.0 + u * (24 if case["optimizer"] == "adam" else 8), "flops": 10.0 * case["ranks"] * n}
    n = case["n"]
    one = n * (5.0 if case.get("dense") else 10.0)          # values (and keys) in, payload out
    back = (n * 1.0 if case.get("dense") else n * 2.0) + 4.0 * case["dim"]
    return {"bytes": one + (back if kind == "codec" else 0.0), "flops": 30.0 * n}


def tolerance(case):
    """Payloads, codes and keys are whole numbers. Floats are sums of fp32 terms in varying order; a value within
    rounding of a bucket border may land in the neighbouring bucket, which the weights see as one quantization step."""
    if case["kind"] in ("encode", "keys"):
        return "exact"
    if case["kind"] in ("codec", "decode"):
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1e-5, "max": 1e-2}
