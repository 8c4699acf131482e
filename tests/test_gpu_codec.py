"""GPU compress / decode kernels against the C++ CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sparse_grad(n, dim, seed, scale=1e-3, positive_only=False):
    rng = np.random.default_rng(seed)
    if dim <= 4 * n or dim < 10_000_000:
        keys = np.sort(rng.choice(dim, n, replace=False)).astype(np.int32)
    else:
        keys = np.unique(rng.integers(0, dim, size=2 * n + 16))
        keys = np.sort(rng.permutation(keys)[:n]).astype(np.int32)
    vals = rng.laplace(0, scale, n).astype(np.float32)
    if positive_only:
        vals = np.abs(vals) + 1e-6
    vals[vals == 0] = 1e-6
    return keys, vals


def _sections(p):
    out = []
    for g in p["groups"]:
        out.append((g["n"], g["col_num"], tuple(g["hash_ids"]), g["table"].tolist() if g["n"] else None,
                    (g["keys"]["num_intervals"], g["keys"]["flag_kind"]) if g["n"] else None,
                    g["keys"]["flag_words"].tolist() if g["n"] else None,
                    g["keys"]["delta_words"].tolist() if g["n"] else None,
                    g.get("restart_raw").tolist() if g["n"] else None))
    return out


@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("n,dim,q,G,rows,ratio", [
    (5000, 200000, 256, 8, 2, 0.3), (1, 1000, 64, 8, 3, 0.2), (2049, 100000000, 128, 1, 3, 0.2),
    (70000, 80000, 256, 8, 2, 0.3), (3000, 2 ** 31 - 2, 300, 4, 1, 0.5), (40000, 5000000, 64, 2, 8, 0.1),
    (300000, 3000000, 256, 8, 3, 0.2)])
def test_payload_bit_exact_with_given_splits(encoder, fused, n, dim, q, G, rows, ratio):
    """Everything downstream of the split points equals the CPU oracle bit for bit, with both key
    encoders (delta_adaptive: the groups' interval counts and flag kinds, the two bit streams and
    the restart points)."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor
    keys, vals = _sparse_grad(n, dim, seed=n)
    qz = oracle.quantile_quantize(vals, q, 128, 1, 2, False)
    splits = qz["splits"].astype(np.float32)
    opts = dict(bin_num=q, group_num=G, row_num=rows, col_ratio=ratio, seed=11, step=7, rank=2, world=4, tie_mode=1,
                key_encoder=1 if encoder == "delta_adaptive" else 0)
    ref = oracle.compress_sparse(keys, vals, dim, opts, splits, float(qz["min"]), float(qz["max"]))
    comp = GpuCompressor(dim, n, q, G, rows, ratio, seed=11, fused=fused, key_encoder=encoder)
    buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=7, rank=2, world=4,
                              given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"]))
    got = comp.payload_bytes(buf)
    pg, pr = oracle.parse(got), oracle.parse(ref)
    for k in ("kind", "step", "rank", "world", "dim", "nnz", "bin_num", "zero_idx", "group_num", "row_num", "col_ratio",
              "key_encoder", "cell_bits", "seed", "restart_interval"):
        assert pg[k] == pr[k], k
    assert np.array_equal(pg["bucket_values"], pr["bucket_values"])
    sg, sr = _sections(pg), _sections(pr)
    for gi, (a, b) in enumerate(zip(sg, sr)):
        for fi, (x, y) in enumerate(zip(a, b)):
            assert x == y, f"group {gi} field {fi} differs"
    kind, k2, v2 = oracle.decompress(got)
    _, k3, v3 = oracle.decompress(ref)
    assert np.array_equal(k2, keys) and np.array_equal(v2, v3)


@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("n,dim,q,G,rows,ratio", [
    (5000, 200000, 256, 8, 2, 0.3), (1, 1000, 64, 8, 3, 0.2), (2049, 100000000, 128, 1, 3, 0.2),
    (3000, 2 ** 31 - 2, 300, 4, 1, 0.5), (300000, 3000000, 256, 8, 3, 0.2)])
def test_huffman_coded_tables(encoder, fused, n, dim, q, G, rows, ratio):
    """cell_bits = 0: the tables travel Huffman-coded. The device's code is canonical and carries restart
    offsets, so its bytes differ from the CPU oracle's tree-walk code; the decoded tables, every other
    section and the decoded gradient are the oracle's bit for bit. The GPU decoder reads both forms."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    keys, vals = _sparse_grad(n, dim, seed=n + 3)
    qz = oracle.quantile_quantize(vals, q, 128, 1, 2, False)
    splits = qz["splits"].astype(np.float32)
    opts = dict(bin_num=q, group_num=G, row_num=rows, col_ratio=ratio, seed=11, step=7, rank=0, world=1, tie_mode=1,
                key_encoder=1 if encoder == "delta_adaptive" else 0, cell_bits=0)
    ref = oracle.compress_sparse(keys, vals, dim, opts, splits, float(qz["min"]), float(qz["max"]))
    comp = GpuCompressor(dim, n, q, G, rows, ratio, seed=11, fused=fused, key_encoder=encoder, cell_bits=0)
    buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=7, rank=0, world=1,
                              given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"]))
    got = comp.payload_bytes(buf)
    pg, pr = oracle.parse(got), oracle.parse(ref)
    assert pg["cell_bits"] == pr["cell_bits"] == 0
    for gi, (a, b) in enumerate(zip(_sections(pg), _sections(pr))):
        for fi, (x, y) in enumerate(zip(a, b)):
            assert x == y, f"group {gi} field {fi} differs"
    _, k2, v2 = oracle.decompress(got)
    _, k3, v3 = oracle.decompress(ref)
    assert np.array_equal(k2, keys) and np.array_equal(v2, v3)
    # with enough cells per group to pay for the code books, the Huffman-coded payload is the smaller one
    plain = GpuCompressor(dim, n, q, G, rows, ratio, seed=11, fused=fused, key_encoder=encoder)
    pb = plain.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=7, rank=0, world=1,
                              given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"]))
    if n >= 100000:
        assert len(got) < len(plain.payload_bytes(pb))
    # both the device-made and the oracle-made payload decode on the GPU to the oracle's values
    want = np.zeros(dim if dim <= 10 ** 8 else 1)
    if dim <= 10 ** 8:
        want[k3] = v3
        dec = GpuDecoder(dim, n, fused=fused)
        out = dec.decode_sum([buf], step=7).cpu().numpy()
        assert np.array_equal(out[k3], v3.astype(np.float32)) and np.count_nonzero(out) <= n
        rb = torch.zeros(max(buf.numel(), len(ref) + 256), dtype=torch.uint8, device="cuda")
        rb[:len(ref)] = torch.frombuffer(bytearray(ref), dtype=torch.uint8).cuda()
        out2 = dec.decode_sum([rb], step=7).cpu().numpy()
        assert np.array_equal(out2, out)


@pytest.mark.parametrize("summary", ["sample", "sketch"])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("n", [100, 255, 256, 257, 2047, 2048, 2049, 4096, 4097, 30000, 1000003])
def test_quantile_splits_rank_error(fused, n, summary):
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor
    dim = max(4 * n, 1000)
    keys, vals = _sparse_grad(n, dim, seed=n + 1)
    q = 256
    comp = GpuCompressor(dim, n, q, 8, 2, 0.3, seed=3, fused=fused, quantile_summary=summary)
    buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda())
    p = oracle.parse(comp.payload_bytes(buf))
    bv = p["bucket_values"]
    assert p["nnz"] == n and 2 <= p["bin_num"] <= q
    assert abs(p["min_value"] - vals.min()) < 1e-12 and abs(p["max_value"] - vals.max()) < 1e-12
    assert np.all(np.diff(bv) > 0)
    # recover the splits from the midpoints and measure their rank error
    splits = np.empty(p["bin_num"] - 1)
    prev = p["min_value"]
    for i in range(p["bin_num"] - 1):
        splits[i] = 2 * float(bv[i]) - prev
        prev = splits[i]
    s = np.sort(vals.astype(np.float64))
    ranks = np.searchsorted(s, splits, side="left") / n
    if n <= 128:
        assert p["bin_num"] >= min(q, n) // 2
    # every split is an order statistic near an even quantile: gaps between consecutive
    # split ranks stay within the k = 128 sketch's error band
    err = np.abs(np.diff(np.concatenate([[0.0], ranks, [1.0]]))).max()
    assert err < 1.0 / q + 0.03, err
    if summary == "sample" and q <= n <= 2048:
        # every value is in the sample: the splits are exact order statistics (the test recovers them from
        # the bucket midpoints in float arithmetic, which can move a rank by one or two)
        assert err <= 1.0 / q + 3.0 / n, err
    kind, k2, v2 = oracle.decompress(comp.payload_bytes(buf))
    assert np.array_equal(k2, keys)
    assert np.all(np.sign(v2) == np.sign(vals)) or (np.sign(v2) != np.sign(vals)).mean() < 0.06


DECODE_MODES = {"staged": dict(fused=False), "fused": dict(fused=True)}


@pytest.mark.parametrize("cell_bits", [-1, 0])
@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
@pytest.mark.parametrize("mode", list(DECODE_MODES))
def test_decode_sum_matches_oracle(mode, encoder, cell_bits):
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim, world = 300000, 3
    fused = mode != "staged"
    comp = GpuCompressor(dim, 20000, 128, 8, 3, 0.2, seed=5, fused=fused, key_encoder=encoder, cell_bits=cell_bits)
    bufs, ref = [], np.zeros(dim)
    for r in range(world):
        keys, vals = _sparse_grad(15000 + 1000 * r, dim, seed=100 + r)
        b = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=4, rank=r, world=world)
        bufs.append(b.clone())
        _, k, v = oracle.decompress(comp.payload_bytes(b))
        ref[k] += v.astype(np.float64) / world
    dec = GpuDecoder(dim, 20000 * world, **DECODE_MODES[mode])
    out = dec.decode_sum(bufs, step=4).cpu().numpy().astype(np.float64)
    assert np.abs(out - ref).max() <= 1e-6 * np.abs(ref).max()
    assert int(dec.acc.abs().max()) == 0
    # a second call gives the same bits (accumulators were left clean, sums are order independent)
    out2 = dec.decode_sum(bufs, step=4).cpu().numpy()
    assert np.array_equal(out2.astype(np.float64), out)


def test_dense_kind_roundtrip_and_mixed_decode():
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim = 50000
    rng = np.random.default_rng(1)
    dense = rng.normal(0, 1e-2, dim).astype(np.float32)
    comp = GpuCompressor(dim, dim, 256, 8, 2, 0.3, seed=1)
    qz = oracle.quantile_quantize(dense, 256, 128, 1, 2, False)
    splits = torch.from_numpy(qz["splits"].astype(np.float32)).cuda()
    b0 = comp.compress_local(None, torch.from_numpy(dense).cuda(), step=2, rank=0, world=2, dense=True,
                             given=(splits, qz["min"], qz["max"])).clone()
    ref0 = oracle.compress_dense(dense, dict(bin_num=256, step=2, rank=0, world=2, seed=1), qz["splits"].astype(np.float32),
                                 float(qz["min"]), float(qz["max"]))
    k0, kk, v0 = oracle.decompress(comp.payload_bytes(b0))
    _, _, vr = oracle.decompress(ref0)
    assert k0 == 2 and np.array_equal(v0, vr)
    # sketch-built splits (no given): decode error bounded by bucket width
    b0s = comp.compress_local(None, torch.from_numpy(dense).cuda(), step=2, rank=0, world=2, dense=True).clone()
    _, _, v0s = oracle.decompress(comp.payload_bytes(b0s))
    assert np.abs(v0s - dense).mean() < 2e-3
    keys, vals = _sparse_grad(4000, dim, seed=8)
    b1 = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=2, rank=1, world=2).clone()
    _, k1, v1 = oracle.decompress(comp.payload_bytes(b1))
    ref = v0s.astype(np.float64) / 2
    ref[k1] += v1.astype(np.float64) / 2
    out = GpuDecoder(dim, dim).decode_sum([b0s, b1], step=2).cpu().numpy()
    assert np.abs(out - ref).max() <= 1e-6 * np.abs(ref).max()


def test_empty_gradient_and_updates():
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim = 10000
    comp = GpuCompressor(dim, 1000, 64, 8, 2, 0.3, seed=2)
    e = comp.compress_local(torch.zeros(0, dtype=torch.int32, device="cuda"), torch.zeros(0, device="cuda"), step=1,
                            rank=0, world=2).clone()
    assert oracle.parse(comp.payload_bytes(e))["kind"] == 0
    keys, vals = _sparse_grad(900, dim, seed=4, scale=1e-1)
    b = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=1, rank=1, world=2).clone()
    _, k, v = oracle.decompress(comp.payload_bytes(b))
    g = np.zeros(dim)
    g[k] = v.astype(np.float64) / 2
    dec = GpuDecoder(dim, 2000)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cap = min(e.numel(), b.numel())
    # SGD
    w = torch.ones(dim, device="cuda")
    dec.decode_update([e.data_ptr(), b.data_ptr()], [None, None], cap, 1, status, w=w, lr=0.5)
    assert int(status.item()) == 0
    assert np.abs(w.cpu().numpy() - (1 - 0.5 * g)).max() < 1e-6
    # lazy Adam: only touched coordinates move
    w = torch.ones(dim, device="cuda")
    m = torch.zeros(dim, device="cuda")
    vv = torch.zeros(dim, device="cuda")
    scale = np.sqrt(1 - 0.999) / (1 - 0.9)
    dec.decode_update([e.data_ptr(), b.data_ptr()], [None, None], cap, 1, status, w=w, lr=0.1, adam_m=m, adam_v=vv,
                      adam_scale=scale)
    mt, vt = 0.1 * g, 0.001 * g * g
    ref = 1 - 0.1 * scale * mt / (np.sqrt(vt) + 1e-8)
    assert np.abs(w.cpu().numpy() - ref).max() < 1e-4
    assert np.abs(m.cpu().numpy() - mt).max() < 1e-7
    untouched = np.ones(dim, bool)
    untouched[k] = False
    assert (w.cpu().numpy()[untouched] == 1).all()


def test_bad_header_and_timeout_are_reported_not_fatal():
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    from sketchml_b200.parallel.failure import PayloadError, StepTimeout, check_status
    dim = 10000
    comp = GpuCompressor(dim, 1000, 64, 8, 2, 0.3, seed=2)
    keys, vals = _sparse_grad(500, dim, seed=4)
    b = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=3).clone()
    dec = GpuDecoder(dim, 1000, budget_s=0.05)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    w = torch.zeros(dim, device="cuda")
    # stale step: the header says 3, the decoder expects 4
    dec.decode_update([b.data_ptr()], [None], b.numel(), 4, status, w=w, lr=1.0)
    with pytest.raises(PayloadError):
        check_status(int(status.item()))
    status.zero_()
    # corrupted header byte -> checksum mismatch
    bad = b.clone()
    bad[40] ^= 0x11
    dec.decode_update([bad.data_ptr()], [None], bad.numel(), 3, status, w=w, lr=1.0)
    with pytest.raises(PayloadError):
        check_status(int(status.item()))
    status.zero_()
    # an arrival flag that nothing sets: the bounded wait gives up and the context stays usable
    flag = torch.zeros(4, dtype=torch.int64, device="cuda")
    dec.decode_update([b.data_ptr()], [flag.data_ptr()], b.numel(), 3, status, w=w, lr=1.0)
    with pytest.raises(StepTimeout):
        check_status(int(status.item()))
    status.zero_()
    dec.reset()
    assert float(w.abs().max()) == 0.0
    flag[0] = 4  # step + 1
    dec.decode_update([b.data_ptr()], [flag.data_ptr()], b.numel(), 3, status, w=w, lr=1.0)
    assert int(status.item()) == 0 and float(w.abs().max()) > 0


def test_non_finite_values_are_reported():
    from sketchml_b200.ops import GpuCompressor
    keys, vals = _sparse_grad(5000, 100000, seed=3)
    vals[17] = -np.inf
    comp = GpuCompressor(100000, 5000, 64, 8, 2, 0.3, seed=1)
    with pytest.raises(RuntimeError, match="invalid kernel input"):
        comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda())
    # the compressor stays usable afterwards
    vals[17] = 1e-3
    comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda())


@pytest.mark.parametrize("bits", [8, 5, 13, 16])
def test_fixed_point_pack_matches_oracle(bits):
    """The pack kernel's code stream against the CPU oracle's BitSet words, and the unpack kernel
    against the oracle's decode (the two norms differ in summation order, so a code may differ by
    one where |v| / norm * max sits on an integer)."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops.baseline_quant import FixedPointCodec
    n, n_max, seed = 100003, 120000, 991
    g = torch.Generator().manual_seed(bits)
    vals = (torch.randn(n_max, generator=g) * 0.01).float()
    keys = torch.sort(torch.randperm(1_000_000, generator=g)[:n_max]).values.int()
    dv, dk = vals.cuda(), keys.cuda()
    cnt = torch.tensor([n], dtype=torch.int64, device="cuda")
    fp = FixedPointCodec(n_max, bits, 1, "cuda")
    fp.pack(dv, cnt, seed)
    out = torch.zeros(n_max, dtype=torch.float32, device="cuda")
    acc = torch.zeros(1_000_000, dtype=torch.float32, device="cuda")
    fp.unpack(dk, fp.codes, fp.norm, cnt, 1, acc=acc, vals_out=out)
    torch.cuda.synchronize()
    code = oracle.fixed_point_encode(vals[:n].double().numpy(), bits, seed)
    assert abs(float(fp.norm.item()) - code["norm"]) <= 1e-12 * code["norm"]
    want = np.asarray(code["words"], dtype=np.uint64).view(np.uint8)
    nbytes = (n * bits + 7) // 8
    got = fp.codes[:nbytes].cpu().numpy()
    assert (got != want[:nbytes]).mean() < 1e-4
    dec = oracle.fixed_point_decode(code)
    step = code["norm"] / ((1 << (bits - 1)) - 1)
    diff = np.abs(out[:n].cpu().numpy().astype(np.float64) - dec)
    assert diff.max() <= step * 1.0001 and (diff > 1e-7 * code["norm"]).mean() < 1e-4
    ref = torch.zeros(1_000_000, dtype=torch.float64)
    ref[keys[:n].long()] = torch.from_numpy(dec)
    assert float((acc.cpu().double() - ref).abs().max()) <= step * 1.0001
    assert float(out[n:].abs().max()) == 0.0


@pytest.mark.parametrize("mode", list(DECODE_MODES))
def test_several_overlapping_payloads_sgd_and_adam(mode):
    """Four payloads with many shared keys: the key-range-owned apply must equal the oracle's
    decoded mean for SGD and one lazy-Adam step on exactly the touched coordinates."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim, P, n = 60000, 4, 9000
    comp = GpuCompressor(dim, n, 128, 8, 3, 0.3, seed=5)
    bufs, g = [], np.zeros(dim)
    for r in range(P):
        keys, vals = _sparse_grad(n - 500 * r, dim // 3, seed=20 + r, scale=1e-2)  # keys crowd the low third: overlaps
        b = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=7, rank=r, world=P).clone()
        _, k, v = oracle.decompress(comp.payload_bytes(b))
        g[k] += v.astype(np.float32).astype(np.float64) / P
        bufs.append(b)
    cap = min(b.numel() for b in bufs)
    ptrs = [b.data_ptr() for b in bufs]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    dec = GpuDecoder(dim, P * n, **DECODE_MODES[mode])
    w = torch.ones(dim, device="cuda")
    dec.decode_update(ptrs, [None] * P, cap, 7, status, w=w, lr=0.5)
    assert int(status.item()) == 0
    assert np.abs(w.cpu().numpy() - (1 - 0.5 * g)).max() < 2e-6
    w = torch.ones(dim, device="cuda")
    m = torch.zeros(dim, device="cuda")
    vv = torch.zeros(dim, device="cuda")
    scale = np.sqrt(1 - 0.999) / (1 - 0.9)
    dec.decode_update(ptrs, [None] * P, cap, 7, status, w=w, lr=0.1, adam_m=m, adam_v=vv, adam_scale=scale)
    assert int(status.item()) == 0
    mt, vt = 0.1 * g, 0.001 * g * g
    ref = 1 - 0.1 * scale * mt / (np.sqrt(vt) + 1e-8)
    touched = g != 0
    assert np.abs(w.cpu().numpy() - ref)[touched].max() < 2e-4
    assert (w.cpu().numpy()[~touched] == 1).all()
    assert np.abs(m.cpu().numpy() - mt).max() < 1e-6
    assert float(dec.acc.abs().max()) == 0  # the accumulators are clean for the next step
    # a second, identical call gives bit-identical results (no order dependence)
    w2 = torch.ones(dim, device="cuda")
    m2 = torch.zeros(dim, device="cuda")
    v2 = torch.zeros(dim, device="cuda")
    dec.decode_update(ptrs, [None] * P, cap, 7, status, w=w2, lr=0.1, adam_m=m2, adam_v=v2, adam_scale=scale)
    assert torch.equal(w, w2) and torch.equal(m, m2) and torch.equal(vv, v2)
    # the packed state layout ({m, v, sum, -} per coordinate) gives the same bits and leaves its sums clean
    quad = torch.zeros((dim, 4), device="cuda")
    w3 = torch.ones(dim, device="cuda")
    dec.decode_update(ptrs, [None] * P, cap, 7, status, w=w3, lr=0.1, adam_m=quad[:, 0], adam_v=quad[:, 1], adam_scale=scale)
    assert int(status.item()) == 0
    assert torch.equal(w, w3) and torch.equal(m, quad[:, 0]) and torch.equal(vv, quad[:, 1])
    assert float(quad[:, 2:].abs().max()) == 0 and float(dec.acc.abs().max()) == 0


@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
def test_decode_skewed_keys_many_ranks(encoder):
    """Eight payloads with Zipf-like keys (many shared coordinates, one nearly empty payload): the fused
    launch must give the bits of the staged launches, which apply the ranks in the same order per
    coordinate, for SGD and for lazy Adam, and the same bits on every repetition."""
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim, P, n = 3_000_000, 8, 40000
    comp = GpuCompressor(dim, n, 256, 8, 3, 0.2, seed=9, key_encoder=encoder)
    rng = np.random.default_rng(5)
    bufs = []
    for r in range(P):
        keys = np.unique(np.minimum(rng.zipf(1.2, 3 * n), dim - 1))[: n - 1000 * r].astype(np.int32)
        if r == 5:
            keys = keys[:3]   # a payload whose groups are nearly all empty
        vals = rng.laplace(0, 1e-2, len(keys)).astype(np.float32)
        bufs.append(comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=3, rank=r, world=P).clone())
    cap = min(b.numel() for b in bufs)
    ptrs = [b.data_ptr() for b in bufs]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref_dec = GpuDecoder(dim, P * n, fused=False)
    w_ref = torch.ones(dim, device="cuda")
    ref_dec.decode_update(ptrs, [None] * P, cap, 3, status, w=w_ref, lr=0.5)
    assert int(status.item()) == 0
    dec = GpuDecoder(dim, P * n, max_groups=8)
    for _ in range(3):
        w = torch.ones(dim, device="cuda")
        dec.decode_update(ptrs, [None] * P, cap, 3, status, w=w, lr=0.5)
        assert int(status.item()) == 0
        assert torch.equal(w, w_ref)

    def adam(d):
        w, m, v = torch.ones(dim, device="cuda"), torch.zeros(dim, device="cuda"), torch.zeros(dim, device="cuda")
        d.decode_update(ptrs, [None] * P, cap, 3, status, w=w, lr=0.1, adam_m=m, adam_v=v, adam_scale=0.3)
        assert int(status.item()) == 0
        return w, m, v
    for a, b in zip(adam(dec), adam(ref_dec)):
        assert torch.equal(a, b)
    quad = torch.zeros((dim, 4), device="cuda")
    wq = torch.ones(dim, device="cuda")
    dec.decode_update(ptrs, [None] * P, cap, 3, status, w=wq, lr=0.1, adam_m=quad[:, 0], adam_v=quad[:, 1], adam_scale=0.3)
    assert int(status.item()) == 0
    for a, b in zip((wq, quad[:, 0], quad[:, 1]), adam(ref_dec)):
        assert torch.equal(a, b)
    assert float(quad[:, 2].abs().max()) == 0
    assert float(dec.acc.abs().max()) == 0


def _key_sets():
    rng = np.random.default_rng(11)
    yield "empty", np.zeros(0, dtype=np.int32)
    yield "single zero", np.array([0], dtype=np.int32)
    yield "single big", np.array([2 ** 31 - 1], dtype=np.int32)
    yield "consecutive", np.arange(5000, dtype=np.int32)
    yield "small gaps", np.cumsum(rng.integers(1, 4, 70001)).astype(np.int32)
    yield "byte gaps", np.cumsum(rng.integers(1, 300, 33333)).astype(np.int32)
    yield "wide gaps", np.sort(rng.choice(2 ** 31 - 2, 20000, replace=False)).astype(np.int32)
    yield "mixed", np.unique(np.concatenate([rng.integers(0, 5000, 3000), rng.integers(0, 2 ** 30, 3000)])).astype(np.int32)
    yield "zipf", np.unique(np.minimum(rng.zipf(1.1, 200000), 50_000_000 - 1)).astype(np.int32)


@pytest.mark.parametrize("name,keys", list(_key_sets()), ids=[n for n, _ in _key_sets()])
def test_delta_adaptive_device_codec_is_bit_exact(name, keys):
    """Device DeltaAdaptive encode equals the CPU oracle word for word; device decode inverts both."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import keys as K
    ref = oracle.delta_adaptive_encode(keys)
    got = K.encode(torch.from_numpy(keys).cuda())
    assert (got.size, got.num_intervals, got.flag_kind) == (ref["size"], ref["num_intervals"], ref["flag_kind"])
    assert (got.flag_bits, got.delta_bits) == (ref["flag_bits"], ref["delta_bits"])
    d = got.to_oracle_dict()
    assert np.array_equal(d["flag_words"], np.asarray(ref["flag_words"], dtype=np.uint64))
    assert np.array_equal(d["delta_words"], np.asarray(ref["delta_words"], dtype=np.uint64))
    assert np.array_equal(oracle.delta_adaptive_decode(d), keys)
    assert np.array_equal(K.decode(got).cpu().numpy(), keys)


def test_delta_adaptive_device_codec_rejects_unsorted_keys():
    from sketchml_b200.ops import keys as K
    with pytest.raises(ValueError):
        K.encode(torch.tensor([1, 5, 5, 9], dtype=torch.int32, device="cuda"))


def _zip_pack(vals, bins):
    from sketchml_b200.ops.baseline_quant import ZipCodec
    n = len(vals)
    zc = ZipCodec(max(n, 1) + 37, bins, 1, "cuda")   # a capacity above n: the padding must not disturb the search
    v = torch.zeros(zc.n_max, device="cuda")
    v[:n] = torch.from_numpy(vals).cuda()
    cnt = torch.tensor([n], dtype=torch.int64, device="cuda")
    zc.pack(v, cnt)
    nb, zero, rounds = (int(x) for x in zc.meta[:3].cpu())
    codes = zc.codes.cpu().numpy()
    codes = codes[:n] if zc.code_bytes == 1 else codes[:2 * n].view(np.uint16)
    return zc, v, cnt, nb, zero, rounds, zc.splits[:max(nb - 1, 0)].cpu().numpy(), zc.mids[:nb].cpu().numpy(), codes.astype(np.int64)


@pytest.mark.parametrize("n,bins", [(1, 16), (2, 2), (3, 2), (77, 8), (1000, 256), (4097, 33), (50001, 256), (300000, 300)])
def test_zipml_device_quantizer_equals_oracle_on_exact_sums(n, bins):
    """Values on a dyadic grid make every prefix sum exact in double, whatever the order of the adds,
    so the device search must pick the very split points of the CPU oracle, round by round."""
    from sketchml_b200.compress import oracle
    rng = np.random.default_rng(n + bins)
    vals = (rng.integers(-2000, 2000, n) / 1024.0).astype(np.float32)
    ref = oracle.zipml_quantize(vals.astype(np.float64), bins)
    zc, v, cnt, nb, zero, rounds, splits, mids, codes = _zip_pack(vals, bins)
    assert nb == ref["bin_num"] and zero == ref["zero_idx"]
    assert np.array_equal(splits.astype(np.float64), ref["splits"])
    assert np.array_equal(mids, ref["values"].astype(np.float32))
    assert np.array_equal(codes, ref["bins"])
    # decode: every value becomes its bucket's midpoint; the accumulating form adds them at the keys
    out = torch.zeros_like(v)
    zc.unpack(None, zc.codes, zc.mids, cnt, 1, vals_out=out)
    assert np.array_equal(out[:n].cpu().numpy(), ref["values"].astype(np.float32)[ref["bins"]])
    keys = torch.from_numpy(np.sort(rng.choice(4 * n + 8, n, replace=False)).astype(np.int32)).cuda()
    kfull = torch.zeros(zc.n_max, dtype=torch.int32, device="cuda")
    kfull[:n] = keys
    acc = torch.zeros(4 * n + 8, device="cuda")
    zc.unpack(kfull, zc.codes, zc.mids, cnt, 1, acc=acc)
    assert torch.equal(acc[keys.long()], out[:n]) and int(torch.count_nonzero(acc)) <= n


@pytest.mark.parametrize("bins", [16, 256])
def test_zipml_device_quantizer_quality_and_empty_input(bins):
    """Real-valued input: the order of the prefix-sum adds differs from the sequential oracle, so near
    ties may fall the other way; the quantization error must still match the oracle's closely."""
    from sketchml_b200.compress import oracle
    _, vals = _sparse_grad(120000, 10 ** 6, seed=5)
    ref = oracle.zipml_quantize(vals.astype(np.float64), bins)
    zc, v, cnt, nb, zero, rounds, splits, mids, codes = _zip_pack(vals, bins)
    assert 2 <= nb <= bins and rounds >= 8 and np.all(np.diff(splits) > 0)
    err_dev = np.mean((mids[codes].astype(np.float64) - vals) ** 2)
    err_ref = np.mean((ref["values"][ref["bins"]] - vals) ** 2)
    assert err_dev <= err_ref * 1.02 + 1e-18, (err_dev, err_ref)
    assert np.all(vals >= np.concatenate([[vals.min()], splits])[codes]) and np.all(vals <= np.concatenate([splits, [vals.max()]])[codes])
    cnt.zero_()
    zc.pack(v, cnt)
    assert int(zc.meta[0]) == 0


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 2047, 2049, 4095, 4096, 4097, 9000, 148 * 32 * 32 + 1])
@pytest.mark.parametrize("q", [2, 64, 256, 1500])
def test_sampled_splits_are_the_sample_s_order_statistics(n, q):
    """The split points of the sample form: the values of rank floor(m (t + 1) / q) of the drawn sample, for
    samples that do not fill the sorted runs, fill them exactly and exceed them, with many equal values too."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, lib as L
    rng = np.random.default_rng(n * 7 + q)
    keys = np.sort(rng.choice(4 * n + 100, n, replace=False)).astype(np.int32)
    for vals in (rng.normal(0, 1e-3, n).astype(np.float32), rng.integers(-3, 4, n).astype(np.float32)):
        comp = GpuCompressor(4 * n + 100, n, q, 8, 2, 0.3, seed=5)
        buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda())
        m = min(n, 4096 if int(L.lib().skml_compress_cluster_size()) == 2 else 2048)
        if n == m:   # (larger inputs: a strided sample whose offset is drawn; checked by the decoded buckets below)
            s = np.sort(vals)
            want = np.unique(s[np.minimum((m * ((np.arange(q - 1) + 1) * (1.0 / q))).astype(np.int64), m - 1)])
            assert np.array_equal(comp.last_splits(), want)
        splits = comp.last_splits()
        got = comp.payload_bytes(buf)
        p = oracle.parse(got)
        assert p["bin_num"] == len(splits) + 1 and p["zero_idx"] == int((splits < 0).sum())
        ref = oracle.compress_sparse(keys, vals, 4 * n + 100, dict(bin_num=q, group_num=8, row_num=2, col_ratio=0.3, seed=5, step=0,
                                     rank=0, world=1, tie_mode=1, key_encoder=0), splits, float(vals.min()), float(vals.max()))
        pr = oracle.parse(ref)
        for a, b in zip(_sections(p), _sections(pr)):
            assert a == b


@pytest.mark.parametrize("n,bins,spread", [
    (16384, 256, 2000), (16385, 257, 2000), (20000, 256, 1), (40000, 8190, 2000), (40000, 4097, 3), (700001, 64, 2000),
    (2500000, 16, 50), (1300001, 2, 2000)])
def test_zipml_split_search_over_its_splits_of_the_work(n, bins, spread):
    """Edges of the split search: the largest search of one block and the smallest of several, keys in registers
    and in memory, few blocks (many kept pairs) and many, and inputs where most errors tie."""
    from sketchml_b200.compress import oracle
    rng = np.random.default_rng(n + bins)
    vals = (rng.integers(-spread, spread + 1, n) / 1024.0).astype(np.float32)   # exact sums, as above
    ref = oracle.zipml_quantize(vals.astype(np.float64), bins)
    zc, v, cnt, nb, zero, rounds, splits, mids, codes = _zip_pack(vals, bins)
    assert nb == ref["bin_num"] and zero == ref["zero_idx"]
    assert np.array_equal(splits.astype(np.float64), ref["splits"])
    assert np.array_equal(mids, ref["values"].astype(np.float32))
    assert np.array_equal(codes, ref["bins"])
    zc.pack(v, cnt)    # the words the blocks share are ready for the next call
    assert int(zc.meta[0]) == nb


@pytest.mark.parametrize("n,bins", [(5000, 16), (16000, 256), (20000, 256), (40000, 16), (120000, 256), (120000, 1000)])
def test_zipml_split_search_on_distinct_errors(n, bins):
    """Continuous values: no two errors of a round tie, and all the largest ones differ by far more than the
    rounding of the prefix sums, so the first rounds must keep exactly the oracle's pairs; later ones may differ
    where a choice hangs on that rounding."""
    from sketchml_b200.compress import oracle
    vals = (np.random.default_rng(n).standard_t(3, n) * 1e-3).astype(np.float32)
    ref = oracle.zipml_quantize(vals.astype(np.float64), bins)
    zc, v, cnt, nb, zero, rounds, splits, mids, codes = _zip_pack(vals, bins)
    same = len(np.intersect1d(splits.astype(np.float64), ref["splits"]))
    assert same >= 0.95 * len(ref["splits"]), (same, len(ref["splits"]))


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 592 * 1024, 592 * 1024 + 1, 1_300_000])
@pytest.mark.parametrize("gaps", ["ones", "mixed", "wide"])
def test_delta_adaptive_device_codec_over_its_runs(n, gaps):
    """Edges of the runs of tiles: less than a tile, exactly one, one run per block full, the first size with two
    tiles a run; fixed and unary flags."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import keys as K
    rng = np.random.default_rng(n)
    d = {"ones": np.ones(n, np.int64), "mixed": np.where(rng.random(n) < 0.9, 1, rng.integers(1, 9000, n)),
         "wide": rng.integers(1, max(2, (2 ** 31 - 2) // n), n)}[gaps]
    keys = np.cumsum(d).astype(np.int32)
    ref = oracle.delta_adaptive_encode(keys)
    got = K.encode(torch.from_numpy(keys).cuda())
    assert (got.num_intervals, got.flag_kind, got.flag_bits, got.delta_bits) == (
        ref["num_intervals"], ref["flag_kind"], ref["flag_bits"], ref["delta_bits"])
    o = got.to_oracle_dict()
    assert np.array_equal(o["flag_words"], np.asarray(ref["flag_words"], dtype=np.uint64))
    assert np.array_equal(o["delta_words"], np.asarray(ref["delta_words"], dtype=np.uint64))
    assert np.array_equal(K.decode(got).cpu().numpy(), keys)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("q,G", [(256, 8), (1500, 20)])
@pytest.mark.parametrize("n", [65, 8 * 1024, 9 * 1024 + 127, 40001])
def test_payload_of_few_blocks_with_long_runs_of_chunks(n, q, G, fused):
    """Two blocks code everything: runs on both sides of four chunks a block, deltas of all widths, more groups than
    three ballots tell apart, more split points than the unrolled part of the search covers."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor
    rng = np.random.default_rng(n + q)
    keys = (np.cumsum(rng.choice([1, 2, 255, 256, 300, 70000], n, p=[.3, .2, .1, .1, .25, .05])) - 1).astype(np.int32)
    dim = int(keys[-1]) + 1
    vals = rng.laplace(0, 1e-3, n).astype(np.float32)
    qz = oracle.quantile_quantize(vals, q, 128, 1, 2, False)
    splits = qz["splits"].astype(np.float32)
    ref = oracle.compress_sparse(keys, vals, dim, dict(bin_num=q, group_num=G, row_num=2, col_ratio=0.3, seed=3, step=1, rank=0,
                                                       world=1, tie_mode=1, key_encoder=0),
                                 splits, float(qz["min"]), float(qz["max"]))
    comp = GpuCompressor(dim, n, q, G, 2, 0.3, seed=3, fused=fused, grid=2)
    buf = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=1, rank=0, world=1,
                              given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"]))
    got = comp.payload_bytes(buf)
    assert _sections(oracle.parse(got)) == _sections(oracle.parse(ref))
    assert np.array_equal(oracle.decompress(got)[2], oracle.decompress(ref)[2])


@pytest.mark.parametrize("q", [2, 256, 300])
@pytest.mark.parametrize("dim", [1, 3, 4, 5, 4099, 50002])
def test_dense_kind_at_ragged_dimensions(dim, q):
    """Codes of one and of two bytes, dimensions on all sides of a multiple of four, against the oracle: whole numbers
    out of the compressor, and a decode of one payload that adds nothing to the bucket values."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dense = np.random.default_rng(dim).normal(0, 1e-2, dim).astype(np.float32)
    qz = oracle.quantile_quantize(dense, q, 128, 1, 2, False)
    splits = qz["splits"].astype(np.float32)
    comp = GpuCompressor(dim, dim, q, 8, 2, 0.3, seed=1)
    buf = comp.compress_local(None, torch.from_numpy(dense).cuda(), step=2, rank=0, world=1, dense=True,
                              given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"])).clone()
    ref = oracle.compress_dense(dense, dict(bin_num=q, step=2, rank=0, world=1, seed=1), splits, float(qz["min"]),
                                float(qz["max"]))
    want = oracle.decompress(ref)[2].astype(np.float32)
    assert np.array_equal(oracle.decompress(comp.payload_bytes(buf))[2].astype(np.float32), want)
    assert np.array_equal(GpuDecoder(dim, dim).decode_sum([buf], step=2).cpu().numpy(), want)


@pytest.mark.parametrize("grid", [0, 2])
@pytest.mark.parametrize("ns", [(1,), (2, 3, 7), (1023, 1025), (9001, 31, 5000, 4098)])
def test_decode_with_exactly_the_keys_it_was_built_for(ns, grid):
    """Lists of every remainder of four at a key capacity of their sum, one chunk to many per block: SGD against the
    oracle's mean (fp32 sums of at most four terms of at most 1e-1: 4 * 2^-24 each, below 1e-7)."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim, P = 30011, len(ns)
    comp = GpuCompressor(dim, max(ns), 64, 8, 3, 0.3, seed=5)
    bufs, g = [], np.zeros(dim)
    for r, n in enumerate(ns):
        keys, vals = _sparse_grad(n, dim, seed=r + n, scale=1e-2)
        vals = np.clip(vals, -0.1, 0.1)
        b = comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=7, rank=r, world=P).clone()
        _, k, v = oracle.decompress(comp.payload_bytes(b))
        g[k] += v.astype(np.float32).astype(np.float64) / P
        bufs.append(b)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(dim, device="cuda")
    dec = GpuDecoder(dim, sum(ns), max_groups=8, grid=grid)
    dec.decode_update([b.data_ptr() for b in bufs], [None] * P, min(b.numel() for b in bufs), 7, status, out_sum=out)
    assert int(status.item()) == 0
    assert np.abs(out.cpu().numpy() - g).max() < 1e-7


@pytest.mark.parametrize("q", [2, 256, 300])
@pytest.mark.parametrize("dim", [1, 5, 4099, 1_000_003, 20_000_001])
def test_dense_kind_with_sampled_splits_into_a_fresh_slot(dim, q):
    """Splits from the kernel's own sample, a buffer that is not zero when it is handed out: every code is the number
    of split points at or below its value, and what lies behind the payload is zero. (A slot cleared beside the code
    pass, without a grid barrier in between, can lose codes of other blocks.)"""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor
    vals = np.random.default_rng(dim).normal(0, 1e-2, dim).astype(np.float32)
    comp = GpuCompressor(dim, dim, q, 8, 2, 0.3, seed=1)
    v = torch.from_numpy(vals).cuda()
    for _ in range(3):
        torch.full((comp.capacity,), 0xA5, dtype=torch.uint8, device="cuda")   # back to the allocator, for the call below
        buf = comp.compress_local(None, v, dense=True)
        p = oracle.parse(comp.payload_bytes(buf))
        want = np.searchsorted(comp.last_splits(), vals, side="right")
        assert p["bin_num"] == len(comp.last_splits()) + 1
        assert np.array_equal(np.asarray(p["dense_codes"][:dim]).astype(np.int64), want)
        assert int(torch.count_nonzero(buf[p["total_bytes"]:])) == 0


@pytest.mark.parametrize("dense", [False, True])
def test_checked_calls_leave_their_results_to_any_stream(dense):
    """`compress_local` and `decode_sum` return when the kernel's last block has reported, not when the kernel has left
    the device: a second stream that waits for nothing reads what the first call's stream would read."""
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim, n = 6_000_000, 6_000_000 if dense else 700_000
    keys, vals = (None, np.random.default_rng(3).normal(0, 1e-2, dim).astype(np.float32)) if dense else _sparse_grad(n, dim, seed=3)
    k, v = None if dense else torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
    comp, dec = GpuCompressor(dim, n, 256, 8, 3, 0.2, seed=2), GpuDecoder(dim, n, max_groups=8)
    want = comp.compress_local(k, v, dense=dense)
    torch.cuda.synchronize()
    want_sum = dec.decode_sum([want]).clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(20):
        buf = comp.compress_local(k, v, dense=dense)
        with torch.cuda.stream(side):
            got = buf.clone()
        out = dec.decode_sum([buf])
        with torch.cuda.stream(side):
            got_sum = out.clone()
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(got_sum, want_sum)


@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
@pytest.mark.parametrize("n,q,G,rows,ratio,levels", [
    (999_999, 256, 8, 3, 0.2, 0), (1_000_000, 256, 8, 3, 0.2, 0), (1_000_003, 64, 20, 1, 0.05, 0),   # around the smallest size
    (1_000_001, 255, 1, 3, 0.1, 0), (1_000_001, 256, 2, 2, 0.3, 0),   # most buckets in a group; one too many
    (1_100_001, 256, 3, 2, 0.001, 0), (1_200_000, 64, 2, 3, 0.45, 0),   # tiny tables; rows of a table in two parts
    (1_200_000, 64, 1, 2, 0.6, 0),                                     # in six: left to the atomics
    (1_000_000, 256, 8, 3, 0.2, 3), (1_000_000, 256, 32, 3, 0.2, 1)])   # few distinct values: empty groups
def test_sketch_inserted_in_shared_memory(n, q, G, rows, ratio, levels, encoder):
    """Large gradients insert into tables in shared memory; the tables equal the oracle's, and the whole payload that of
    the staged launches, which insert with atomics."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import GpuCompressor
    dim = 3 * n
    keys, vals = _sparse_grad(n, dim, seed=n + q)
    if levels:
        vals = (np.arange(n) % levels + 1).astype(np.float32) * np.where(np.arange(n) % 5 < 2, -1, 1).astype(np.float32)
    kt, vt = torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
    comps = [GpuCompressor(dim, n, q, G, rows, ratio, seed=11, fused=fused, key_encoder=encoder) for fused in (True, False)]
    own = [c.payload_bytes(c.compress_local(kt, vt, step=3)) for c in comps]
    assert own[0] == own[1]
    qz = oracle.quantile_quantize(vals, q, 128, 1, 2, False)
    splits = qz["splits"].astype(np.float32)
    opts = dict(bin_num=q, group_num=G, row_num=rows, col_ratio=ratio, seed=11, step=7, rank=0, world=1, tie_mode=1,
                key_encoder=1 if encoder == "delta_adaptive" else 0)
    ref = oracle.parse(oracle.compress_sparse(keys, vals, dim, opts, splits, float(qz["min"]), float(qz["max"])))
    buf = comps[0].compress_local(kt, vt, step=7, given=(torch.from_numpy(splits).cuda(), qz["min"], qz["max"]))
    got = oracle.parse(comps[0].payload_bytes(buf))
    for gi, (a, b) in enumerate(zip(_sections(got), _sections(ref))):
        for fi, (x, y) in enumerate(zip(a, b)):
            assert x == y, f"group {gi} field {fi} differs"


@pytest.mark.parametrize("n", [8191, 8192, 8193, 148 * 8192, 148 * 8192 + 1, 2_500_003])
@pytest.mark.parametrize("gaps", ["ones", "mixed", "wide"])
def test_delta_adaptive_device_codec_over_tiles_and_runs(n, gaps):
    """Less than a tile, one tile, the first bits of a second run; one tile a run everywhere, then several. A list that
    does not start on 16 bytes gives the same code."""
    from sketchml_b200.compress import oracle
    from sketchml_b200.ops import keys as K
    rng = np.random.default_rng(n)
    d = {"ones": np.ones(n, np.int64), "mixed": np.where(rng.random(n) < 0.9, 1, rng.integers(1, 700, n)),
         "wide": rng.integers(1, max(2, (2 ** 31 - 2) // n), n)}[gaps]
    keys = np.cumsum(d).astype(np.int32)
    ref = oracle.delta_adaptive_encode(keys)
    room = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    room[1:] = torch.from_numpy(keys).cuda()
    for t in (torch.from_numpy(keys).cuda(), room[1:]):
        got = K.encode(t)
        assert (got.num_intervals, got.flag_kind, got.flag_bits, got.delta_bits) == (
            ref["num_intervals"], ref["flag_kind"], ref["flag_bits"], ref["delta_bits"])
        o = got.to_oracle_dict()
        assert np.array_equal(o["flag_words"], np.asarray(ref["flag_words"], dtype=np.uint64))
        assert np.array_equal(o["delta_words"], np.asarray(ref["delta_words"], dtype=np.uint64))
        assert np.array_equal(K.decode(got).cpu().numpy(), keys)


@pytest.mark.parametrize("n", [4059, 4060, 16384 + 5, 148 * 4096 - 37, 148 * 4096 - 36, 148 * 8192 - 37, 148 * 8192 - 36])
def test_zipml_sort_over_its_blocks(n):
    """One block, two, a ragged slice, every block with four and then more values a thread, the largest size and the first
    beyond it (values on a dyadic grid: the search must pick the oracle's very split points; signed zeros among them)."""
    from sketchml_b200.compress import oracle
    rng = np.random.default_rng(n)
    vals = (rng.integers(-30000, 30000, n) / 1024.0).astype(np.float32)
    vals[rng.random(n) < 0.01] *= 0.0      # both zeros
    ref = oracle.zipml_quantize(vals.astype(np.float64), 256)
    _, _, _, nb, zero, _, splits, mids, codes = _zip_pack(vals, 256)
    assert nb == ref["bin_num"] and zero == ref["zero_idx"]
    assert np.array_equal(splits.astype(np.float64), ref["splits"])
    assert np.array_equal(mids, ref["values"].astype(np.float32)) and np.array_equal(codes, ref["bins"])


@pytest.mark.parametrize("n", [8192, 8193, 500_001, 148 * 8192])
def test_key_decode_whose_blocks_stop_waiting_gives_the_keys(n):
    """No caller looks at a decode's status: where its blocks' wait for one another runs out (here: at once), the keys
    come out all the same, never a mark in the place of one."""
    from sketchml_b200.ops import keys as K
    from sketchml_b200.ops import lib as L
    d = np.random.default_rng(n).integers(1, (2 ** 31 - 2) // n, n)
    keys = torch.from_numpy(np.cumsum(d).astype(np.int32)).cuda()
    e = K.encode(keys)
    assert e.flag_kind == 0        # (blocks wait for one another)
    for budget in (1, 3000):    # cycles: every block gives up at the first barrier, or some at either
        work, out = K._workspace(keys.device), torch.full((n,), -7, dtype=torch.int32, device="cuda")
        L.check(L.lib().skml_da_decode(e.flag_words.data_ptr(), e.flag_words.numel(), e.delta_words.data_ptr(), e.delta_words.numel(), n,
                                       e.num_intervals, e.flag_kind, e.flag_bits, work.data_ptr(), None, out.data_ptr(), budget,
                                       L.stream()), "skml_da_decode")
        assert torch.equal(out, keys)


@pytest.mark.parametrize("n", [8192, 8193, 100_000, 148 * 8192, 148 * 8192 + 1])
def test_a_fault_in_any_run_of_keys_is_every_blocks(n):
    """The fault travels with the run's counts: no block goes on, wherever it lies (borders of runs too), and the call
    after it, in the same memory, is not touched by it."""
    from sketchml_b200.ops import keys as K
    keys = torch.arange(0, 3 * n, 3, dtype=torch.int32, device="cuda")
    for at in sorted({1, 8191, min(8192, n - 1), n // 2, n - 1}):
        bad = keys.clone()
        bad[at] = bad[at - 1]
        with pytest.raises(ValueError):
            K.encode(bad)
        assert torch.equal(K.decode(K.encode(keys)), keys)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_key_codec_on_every_device_of_a_process():
    """The encoder's shared memory is above what a kernel gets unasked, and the limit is set for one device only."""
    from sketchml_b200.ops import keys as K
    keys = torch.arange(0, 60000, 3, dtype=torch.int32)
    for d in (0, 1, 0):
        with torch.cuda.device(d):
            e = K.encode(keys.to(f"cuda:{d}"))
            assert torch.equal(K.decode(e).cpu(), keys)


@pytest.mark.parametrize("n", [1, 40_000, 300_000, 20_000_000])
@pytest.mark.parametrize("gap", [1, 100])
def test_key_code_holds_no_more_memory_than_twice_its_length(n, gap):
    """The streams' buffer is their length, twice that or 256 KB more at most; a long list is never given room that its
    code does not need, not even for the length of the call."""
    from sketchml_b200.ops import keys as K
    keys = torch.arange(0, gap * n, gap, dtype=torch.int32, device="cuda")
    K.decode(K.encode(keys[:8]))                # (the pinned words)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    e = K.encode(keys)
    used = 8 * (e.flag_words.numel() + e.delta_words.numel())
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in (e.flag_words, e.delta_words)}
    assert sum(held.values()) <= max(2 * used, used + (256 << 10))
    if n > 14_000_000:
        assert torch.cuda.max_memory_allocated() - before <= used + (1 << 20)
    assert torch.equal(K.decode(e), keys)


def test_key_encode_does_not_leave_its_room():
    from sketchml_b200.ops import keys as K
    from sketchml_b200.ops import lib as L
    keys = torch.arange(0, 300_000, 3, dtype=torch.int32, device="cuda")
    e = K.encode(keys)
    cs, need = K._call_state(), e.flag_words.numel() + e.delta_words.numel()
    for room, ok in ((need, True), (need - 1, False)):
        out, work = torch.full((need + 8,), -1, dtype=torch.int64, device="cuda"), K._workspace(keys.device)
        L.check(L.lib().skml_da_encode(keys.data_ptr(), keys.numel(), work.data_ptr(), out.data_ptr(), room, 0, cs.words.data_ptr(), cs.status_ref,
                                       L.stream()), "skml_da_encode")
        assert (cs.status.value == 0) == ok and bool((out[need if ok else 0:] == -1).all())
        if ok:
            assert torch.equal(out[:need], torch.cat([e.flag_words, e.delta_words]))


@pytest.mark.parametrize("n,n_max,bound,in_shared", [
    (1_300_000, 1_300_000, 0, False), (1_300_000, 3_999_999, 0, False), (1_300_000, 4_000_000, 0, True),   # room alone says little
    (1_249_999, 4_000_000, 0, False), (1_300_000, 1_400_000, 1_300_000, True), (1_300_000, 2_000_000, 1_400_000, True)])
def test_where_the_sketch_is_inserted_when_the_number_of_keys_is_on_the_device(n, n_max, bound, in_shared):
    """Room for 1M keys does not choose the kernel that inserts in shared memory, which costs launches of fewer keys 3 us
    and more; a known number does. The payload is the same either way."""
    import ctypes
    from sketchml_b200.ops import GpuCompressor
    from sketchml_b200.ops import lib as L
    dim = 3 * n
    keys, vals = _sparse_grad(n, dim, seed=n)
    kt, vt = torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
    comp, known = (GpuCompressor(dim, m, 256, 8, 3, 0.2, seed=11) for m in (n_max, n))
    buf = torch.zeros(comp.capacity, dtype=torch.uint8, device="cuda")
    meta, status = torch.tensor([n, 1, 0, 0], dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    a = comp.make_args(kt, vt, meta, 3, 0, 1, buf.data_ptr(), buf.numel(), [buf.data_ptr()], [None], status, None, None)
    a.n_bound = bound
    L.check(L.lib().skml_compress_sparse(ctypes.byref(a), L.stream()), "skml_compress_sparse")
    assert int(status) == 0
    assert (int(comp.workspace[:256].view(torch.int64)[15]) != 0) == in_shared       # the stage's time stamp
    assert comp.payload_bytes(buf) == known.payload_bytes(known.compress_local(kt, vt, step=3))


def test_settings_changed_after_a_workspace_of_the_least_size():
    """A compressor made for Huffman-coded tables has no room for the insert in shared memory: with plain tables set
    afterwards it inserts with atomics, the payload being the same."""
    from sketchml_b200.ops import GpuCompressor
    n, dim = 1_400_000, 4_000_000
    keys, vals = _sparse_grad(n, dim, seed=5)
    kt, vt = torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
    c, plain = GpuCompressor(dim, n, 256, 8, 3, 0.2, seed=11, cell_bits=0), GpuCompressor(dim, n, 256, 8, 3, 0.2, seed=11)
    c.compress_local(kt, vt, step=3)
    assert c.ws_bytes < plain.ws_bytes - n
    c.cell_bits = -1
    assert c.payload_bytes(c.compress_local(kt, vt, step=3)) == plain.payload_bytes(plain.compress_local(kt, vt, step=3))


@pytest.mark.parametrize("encoder", ["delta_binary", "delta_adaptive"])
@pytest.mark.parametrize("n,q,G,rows,ratio,levels,in_shared", [
    (1_249_999, 256, 8, 3, 0.2, 0, False), (1_250_000, 256, 8, 3, 0.2, 0, True), (1_250_003, 64, 20, 3, 0.05, 0, False),   # the fewest keys, more
    (2_000_003, 64, 20, 3, 0.05, 0, True), (2_499_999, 256, 8, 2, 0.1, 0, False), (2_500_001, 256, 8, 2, 0.1, 0, True),    # for many groups, fewer rows
    (6_000_001, 255, 8, 1, 0.05, 0, True), (2_600_000, 255, 1, 3, 0.04, 0, True), (2_600_000, 256, 2, 3, 0.08, 0, False),  # most buckets in a group; one too many
    (1_300_001, 256, 3, 3, 0.001, 0, True), (2_900_000, 128, 8, 3, 0.6, 0, False), (3_100_000, 128, 8, 3, 0.6, 0, True),   # tiny tables; rows in two parts
    (4_100_001, 128, 8, 3, 0.7, 0, True), (4_100_000, 128, 8, 3, 0.95, 0, False),                                         # in three; in four
    (1_300_000, 256, 8, 3, 0.2, 3, True), (1_300_000, 256, 32, 3, 0.2, 1, False), (2_100_000, 256, 20, 3, 0.2, 1, False)])  # few distinct values: empty groups, one of many parts
def test_large_gradients_insert_where_it_pays(n, q, G, rows, ratio, levels, in_shared, encoder):
    """Where the sketch is inserted (the stage of its own leaves a time stamp), and that the payload is that of the staged
    launches, which insert with atomics, byte for byte."""
    from sketchml_b200.ops import GpuCompressor
    dim = 3 * n
    g = torch.Generator(device="cuda").manual_seed(n + q)
    kt = torch.cumsum(torch.randint(1, 4, (n,), generator=g, device="cuda"), 0).to(torch.int32) - 1
    vt = torch.randn(n, generator=g, device="cuda") * 1e-3
    if levels:
        i = torch.arange(n, device="cuda")
        vt = (i % levels + 1).float() * torch.where(i % 5 < 2, -1.0, 1.0)
    comps = [GpuCompressor(dim, n, q, G, rows, ratio, seed=11, fused=fused, key_encoder=encoder) for fused in (True, False)]
    own = [c.payload_bytes(c.compress_local(kt, vt, step=3)) for c in comps]
    assert own[0] == own[1]
    assert (int(comps[0].workspace[:256].view(torch.int64)[15]) != 0) == in_shared


@pytest.mark.parametrize("P,n,blocks", [(2, 1000, 1), (2, 1024, 1), (2, 1025, 1), (2, 1280, 1), (2, 1281, 1), (3, 5000, 2), (3, 9000, 3), (2, 3000, 0)])
def test_decode_passes_of_one_and_of_several_iterations(P, n, blocks):
    """A block's slice of a rank's keys in one iteration of 1024 entries, at its edge, in one and a little (up to 1280), and in
    several: the bits of the staged launches, for SGD and for lazy Adam."""
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    dim = 4 * n
    comp = GpuCompressor(dim, n, 64, 4, 2, 0.3, seed=9)
    bufs = []
    for r in range(P):
        m = n if r < 2 else n // 5       # the last rank's pass is a short one behind long ones
        keys, vals = _sparse_grad(m, dim, seed=100 * n + r)
        bufs.append(comp.compress_local(torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda(), step=3, rank=r, world=P).clone())
    ptrs, cap, status = [b.data_ptr() for b in bufs], min(b.numel() for b in bufs), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for dec in (GpuDecoder(dim, P * n, fused=False), GpuDecoder(dim, P * n, max_groups=4, grid=blocks)):
        w = torch.ones(dim, device="cuda")
        dec.decode_update(ptrs, [None] * P, cap, 3, status, w=w, lr=0.5)
        wa, m, v = torch.ones(dim, device="cuda"), torch.zeros(dim, device="cuda"), torch.zeros(dim, device="cuda")
        dec.decode_update(ptrs, [None] * P, cap, 3, status, w=wa, lr=0.1, adam_m=m, adam_v=v, adam_scale=0.3)
        assert int(status.item()) == 0
        out.append((w, wa, m, v))
    assert all(torch.equal(a, b) for a, b in zip(*out)) and int((out[0][0] != 1).sum()) > n // 2


@pytest.mark.parametrize("n", [700, 1024, 1025, 3000, 6107, 6108])
def test_zipml_sort_of_one_block(n):
    """Values that stay in shared memory between the passes, up to the largest size and the first beyond it (37 values of
    room more than there are): the oracle's split points, both zeros among the values."""
    from sketchml_b200.compress import oracle
    rng = np.random.default_rng(n)
    vals = (rng.integers(-30000, 30000, n) / 1024.0).astype(np.float32)
    vals[rng.random(n) < 0.01] *= 0.0
    ref = oracle.zipml_quantize(vals.astype(np.float64), 64)
    _, _, _, nb, zero, _, splits, mids, codes = _zip_pack(vals, 64)
    assert nb == ref["bin_num"] and zero == ref["zero_idx"]
    assert np.array_equal(splits.astype(np.float64), ref["splits"])
    assert np.array_equal(mids, ref["values"].astype(np.float32)) and np.array_equal(codes, ref["bins"])


def test_launches_of_all_kinds_share_a_workspace():
    """A launch takes one of two sets of control words and opens the other for the next one: sparse, dense, empty and staged
    launches in any order leave what they leave in a fresh workspace."""
    from sketchml_b200.ops import GpuCompressor
    dim, n = 60_000, 50_000
    new = lambda fused=True: GpuCompressor(dim, n, 64, 4, 2, 0.3, seed=9, fused=fused)
    comp = new()
    g = torch.Generator(device="cuda").manual_seed(3)
    for i, what in enumerate(["sparse", "dense", "sparse", "empty", "sparse", "sparse", "staged", "sparse", "staged", "dense", "dense", "empty", "staged", "sparse"]):
        if what == "dense":
            keys, vals, kind = None, torch.randn(dim, generator=g, device="cuda"), dict(dense=True)
        else:
            m = 0 if what == "empty" else (n if i % 2 else 777)
            keys = torch.randperm(dim, generator=g, device="cuda")[:m].sort().values.int()
            vals, kind = torch.randn(m, generator=g, device="cuda") * 10.0 ** -i, {}
        comp.fused = what != "staged"
        got = comp.compress_local(keys, vals, step=i, **kind)
        assert torch.equal(got, new(comp.fused).compress_local(keys, vals, step=i, **kind)), (i, what)


@pytest.mark.parametrize("n,dim", [(1, 5), (5000, 50_000), (148 * 1024 - 8 * 1024, 1_000_000), (148 * 1024 - 8 * 1024 + 1, 1_000_000), (60_000, 60_000)])
def test_decode_of_few_keys_by_a_block_per_sm(n, dim):
    """Either side of the limit (room for a chunk per SM and one per group), a dense payload too: the bits of three blocks an SM."""
    from sketchml_b200.ops import GpuCompressor, GpuDecoder
    g = torch.Generator(device="cuda").manual_seed(n)
    dense = n == dim
    keys = None if dense else torch.randperm(dim, generator=g, device="cuda")[:n].sort().values.int()
    vals = torch.randn(n, generator=g, device="cuda")
    buf = GpuCompressor(dim, n, 64, 8, 2, 0.3, seed=5).compress_local(keys, vals, dense=dense)
    status, out = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for grid in (0, 3 * torch.cuda.get_device_properties(0).multi_processor_count):
        dec = GpuDecoder(dim, n, max_groups=8, grid=grid)
        w, sumsq, reg = torch.ones(dim, device="cuda"), torch.full((1,), float(dim), dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
        dec.track_norm(sumsq, reg, 0.5)
        dec.decode_update([buf.data_ptr()], [None], buf.numel(), 0, status, w=w, lr=0.5)
        assert int(status.item()) == 0 and int((w != 1).sum()) > n // 2
        norm = float(w.double().norm())
        # n changes of a squared weight in fp32, each within 2^-22 of itself
        assert abs(float(reg) - 0.5 * norm) <= 1e-6 * norm and abs(float(sumsq) - norm * norm) <= 2e-6 * norm * norm
        out.append((w, dec.decode_sum([buf])))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("n,bins", [(1535, 64), (1536, 64), (1537, 64), (1538, 2), (3071, 256), (3072, 1500), (3073, 1535), (6200, 1537), (16385, 700)])
def test_zipml_last_rounds_around_their_room(n, bins):
    """Searches whose rounds reach the 1,536 candidates of the last rounds from the start, exactly, one above, or never; odd numbers."""
    from sketchml_b200.compress import oracle
    vals = (np.random.default_rng(n + bins).integers(-3000, 3001, n) / 1024.0).astype(np.float32)   # exact sums
    ref = oracle.zipml_quantize(vals.astype(np.float64), bins)
    zc, v, cnt, nb, zero, rounds, splits, mids, codes = _zip_pack(vals, bins)
    assert nb == ref["bin_num"] and zero == ref["zero_idx"] and np.array_equal(splits.astype(np.float64), ref["splits"])
    assert np.array_equal(mids, ref["values"].astype(np.float32)) and np.array_equal(codes, ref["bins"])
