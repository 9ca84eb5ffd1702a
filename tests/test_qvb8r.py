"""QVB8R (entropy-coded QVB8): the synthetic encoder against the oracle decoder, the container round trip, and the
CUDA kernels against the oracle on seeded packs.  The oracle decoder, the encoder, the container code and the kernels
are pinned on files written and decoded by the reference itself in tests/test_qvb8r_golden.py."""
import numpy as np
import pytest
import torch

import oracle
from qvb8_b200 import packs, rans, synth

DEV = "cuda:0"
TOL = 1e-2
TIGHT = 2e-5


def _pack(Q, P, seed, K=3, T=None, tau=2e-3):
    W = synth.synth_weight(Q, P, seed)
    return W, synth.encode_qvb8r(W, tau=tau, K=K, T=T)


def _dense(d):
    """fp32 restored weights with the exact escapes written over (what a dense reader produces)."""
    return oracle.qvb8r_dense(d)


def test_encoder_roundtrip_and_certificate():
    W, d = _pack(80, 256, seed=11, K=3, T=4)
    tab = rans.slot_tables(d["freq"])
    assert np.array_equal(tab, oracle.slot_tables(d["freq"]))
    assert int(d["freq"].astype(np.int64).sum(1).min()) == 4096 and int(d["freq"].max()) <= 1024
    words = np.concatenate([d["words"], np.zeros(rans.PAD_WORDS, np.uint32)])
    ids = oracle.rans_decode_ids(words, d["tile_off"].astype(np.int64), d["states"], d["tiles"].astype(np.int64), tab,
                                 d["perm"], d["drow"].astype(np.int32), 80, 256)
    band = oracle.rans_restore_f32(ids, d["min_s"], d["tau_s"])
    Wd = _dense(d)
    # every weight within tau of the source after the fp16 rounding the certificate is stated on
    err = np.abs(Wd.astype(np.float16).astype(np.float64) - W.float().numpy().astype(np.float64))
    assert float(err.max()) <= 2e-3
    # the stored differences are exact - band at the escaped positions
    ei = d["esc_idx"]
    assert np.array_equal((d["esc_val"] - band.reshape(-1)[ei]).astype(np.float32), d["esc_delta"])
    assert d["words"].size * 32 / (80 * 256) < 8.0       # it does compress


def test_container_roundtrip():
    _, d = _pack(48, 128, seed=5, K=2, T=8)
    blob = packs.write_qvb8r(d, Q=d["Q"], P=d["P"], min_s=d["min_s"], tau_s=d["tau_s"], esc_idx=d["esc_idx"],
                             esc_val=d["esc_val"], esc_delta=d["esc_delta"], cert=dict(tau=d["tau"], max_err=d["max_err"]))
    r = packs.read_qvb8r(blob)
    for k in ("perm", "freq", "tiles", "tile_off", "states", "words", "drow", "min_s", "tau_s", "esc_idx", "esc_val", "esc_delta"):
        assert np.array_equal(np.asarray(r[k]), np.asarray(d[k]).astype(np.asarray(r[k]).dtype)), k
    assert np.array_equal(_dense(r).view(np.uint32), _dense(d).view(np.uint32))
    bad = bytearray(blob); bad[200] ^= 1
    with pytest.raises(packs.PackFormatError):
        packs.read_qvb8r(bytes(bad))


def test_blocks_schedule():
    tiles = np.array([[0, 0, 4]] * 10 + [[1, 40, 4]] * 3, np.int64)
    b = rans.blocks_for(tiles, 8)
    assert b.tolist() == [[0, 0, 8], [0, 8, 2], [1, 10, 3]]


@pytest.mark.gpu
@pytest.mark.parametrize("Q,P,K,T", [(80, 256, 3, 4), (300, 1024, 2, 1), (64, 4096, 1, 8), (1000, 512, 4, 3)])
def test_gpu_ids_and_decode(cuda_lib, Q, P, K, T):
    from qvb8_b200.ext_qvb8r import core_tensors, ext
    _, d = _pack(Q, P, seed=Q + P, K=K, T=T)
    core = core_tensors(d, DEV)
    tab = rans.slot_tables(d["freq"])
    words = np.concatenate([d["words"], np.zeros(rans.PAD_WORDS, np.uint32)])
    want_ids = oracle.rans_decode_ids(words, d["tile_off"].astype(np.int64), d["states"], d["tiles"].astype(np.int64), tab,
                                      d["perm"], d["drow"].astype(np.int32), Q, P)
    got = ext.ids(P, *core)
    assert np.array_equal(got.cpu().numpy(), want_ids)                       # bit-exact
    band = oracle.rans_restore_f32(want_ids, d["min_s"], d["tau_s"])
    nblk = core[4].numel() // 3
    for code, dt, ref in ((2, torch.float32, band),
                          (0, torch.float16, torch.from_numpy(band).to(torch.float16).numpy()),
                          (1, torch.bfloat16, None)):
        Wg = ext.decode(*core, P, code, 0, nblk, -1, 0)
        assert Wg.dtype == dt
        if ref is None:
            assert torch.equal(Wg.cpu(), torch.from_numpy(band).to(torch.bfloat16))
        else:
            assert np.array_equal(Wg.cpu().numpy().view(np.uint16 if code == 0 else np.uint32),
                                  ref.view(np.uint16 if code == 0 else np.uint32))
    # a block range as a compact chunk in sorted order
    b0, nb = nblk // 3, max(1, nblk // 2)
    blocks = core[4].cpu().numpy().reshape(-1, 3)
    tiles = np.asarray(d["tiles"]).reshape(-1, 3)
    t_first, t_last = blocks[b0][1], blocks[b0 + nb - 1][1] + blocks[b0 + nb - 1][2] - 1
    row_base = int(tiles[t_first][1]); nrows = int(tiles[t_last][1] + tiles[t_last][2]) - row_base
    chunk = ext.decode(*core, P, 2, b0, nb, row_base, nrows)
    want_chunk = band[np.asarray(d["perm"])[row_base:row_base + nrows]]
    assert np.array_equal(chunk.cpu().numpy().view(np.uint32), want_chunk.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 3, 8, 13])
def test_gpu_products(cuda_lib, M):
    from qvb8_b200.ext_qvb8r import core_tensors, escape_csr, ext
    Q, P = 260, 1024
    _, d = _pack(Q, P, seed=70 + M, K=3, T=2)
    core = core_tensors(d, DEV)
    Wd = _dense(d)                                                           # exact escapes written over
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.float32)
    want = oracle.matmul_f32w(X.cpu().numpy(), Wd, narrow_x=False)
    if M == 1:
        y = ext.gemv(X.reshape(-1), *core).reshape(1, -1)
    elif M <= 8:
        y = ext.multi(X, *core)
        yb = ext.multi(X.to(torch.bfloat16), *core)                           # bf16 X is exact in fp32
        ext.fix_escapes(X.to(torch.bfloat16).float(), *escape_csr(d, DEV), yb)
        wb = oracle.matmul_f32w(X.to(torch.bfloat16).float().cpu().numpy(), Wd, narrow_x=False)
        assert np.linalg.norm(yb.cpu().numpy() - wb) / np.linalg.norm(wb) < TIGHT
    else:
        y = None
    if y is not None:
        ext.fix_escapes(X, *escape_csr(d, DEV), y)
        err = np.linalg.norm(y.cpu().numpy() - want) / np.linalg.norm(want)
        assert err < TOL and err < TIGHT, err
    # tensor-core contract: band rounded once to fp16, fp16 X
    Xh = X.to(torch.float16)
    yt = ext.tc(Xh, *core, 8)
    ids = oracle.rans_decode_ids(np.concatenate([d["words"], np.zeros(rans.PAD_WORDS, np.uint32)]),
                                 d["tile_off"].astype(np.int64), d["states"], d["tiles"].astype(np.int64),
                                 rans.slot_tables(d["freq"]), d["perm"], d["drow"].astype(np.int32), Q, P)
    W16 = oracle.rans_restore_f32(ids, d["min_s"], d["tau_s"]).astype(np.float16).astype(np.float32)
    wt = oracle.matmul_f32w(Xh.float().cpu().numpy(), W16, narrow_x=False)
    errt = np.linalg.norm(yt.cpu().numpy() - wt) / np.linalg.norm(wt)
    assert errt < TOL and errt < TIGHT, errt
    assert torch.equal(yt, ext.tc(Xh, *core, 8))                              # fixed summation order


def test_linear_module_builds_on_cpu_and_chunks_cover_all_rows():
    """Host-side logic of the module: buffers, escape CSR, chunk plan (no kernel call)."""
    from qvb8_b200.linear_r import QVBandLinearV8R, plan_chunks
    _, d = _pack(100, 256, seed=21, K=3, T=4)
    mod = QVBandLinearV8R(d, device="cpu")
    assert mod.whole and len(mod.chunks) == 1 and mod.chunks[0].rows == 100
    assert sorted(mod.chunk_rows.tolist()) == list(range(100))
    assert int(mod.esc_ptr[-1]) == len(d["esc_idx"]) == mod.esc_delta16.numel()
    small = type("Small", (QVBandLinearV8R,), {"CHUNK_BYTES": 2 * 256 * 16})     # 16 rows of fp16 per chunk
    m2 = small(d, device="cpu")
    assert len(m2.chunks) > 1 and not m2.whole
    assert sum(c.rows for c in m2.chunks) == 100 and m2.chunks[-1].esc1 == m2.chunk_esc_pos.numel() == len(d["esc_idx"])
    assert all(a.row0 + a.rows == b.row0 and a.block0 + a.nblocks == b.block0 for a, b in zip(m2.chunks, m2.chunks[1:]))
    # every chunk escape lands on the element it names: sorted row (row0 + pos // P) is original row chunk_rows[...]
    P = 256
    got = set()
    for c in m2.chunks:
        for pos in m2.chunk_esc_pos[c.esc0:c.esc1].tolist():
            assert 0 <= pos < c.rows * P
            got.add(int(m2.chunk_rows[c.row0 + pos // P]) * P + pos % P)
    assert got == set(int(v) for v in d["esc_idx"])
    tiles = np.array([[0, 0, 4], [0, 4, 4], [0, 8, 4], [1, 12, 2], [1, 14, 2]], np.int64)
    blocks = rans.blocks_for(tiles, 2)
    assert plan_chunks(tiles, blocks, 8) == [(0, 1, 0, 8), (1, 2, 8, 8)]
    assert plan_chunks(tiles, blocks, 1) == [(0, 1, 0, 8), (1, 1, 8, 4), (2, 1, 12, 4)]
    mod.to(torch.bfloat16)
    assert mod.min_s.dtype == torch.float32 and mod.esc_delta.dtype == torch.float32


@pytest.mark.gpu
@pytest.mark.parametrize("M,chunk_rows", [(1, None), (5, None), (12, None), (40, None), (130, None), (130, 32)])
def test_linear_module_forward(cuda_lib, M, chunk_rows):
    from qvb8_b200.linear_r import QVBandLinearV8R
    Q, P = 260, 1024
    _, d = _pack(Q, P, seed=31, K=3, T=2)
    cls = QVBandLinearV8R if chunk_rows is None else type("Small", (QVBandLinearV8R,), {"CHUNK_BYTES": 2 * P * chunk_rows})
    bias = torch.linspace(-1, 1, Q)
    mod = cls(d, bias=bias, device=DEV)
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.bfloat16)
    y = mod(X.reshape(1, M, P))
    assert y.shape == (1, M, Q) and y.dtype == torch.bfloat16
    want = oracle.matmul_f32w(X.float().cpu().numpy(), _dense(d), narrow_x=False) + bias.numpy()[None, :]
    err = np.linalg.norm(y.float().cpu().numpy().reshape(M, Q) - want) / np.linalg.norm(want)
    assert err < TOL, err                                 # bf16 output rounding: ~2e-3
    yf = mod(X.float())
    errf = np.linalg.norm(yf.cpu().numpy() - want) / np.linalg.norm(want)
    assert errf < 1e-3, errf                             # fp16 weight rounding above 8 rows
    Wd = mod.dense(torch.float32)
    assert np.array_equal(Wd.cpu().numpy().view(np.uint32), _dense(d).view(np.uint32))


def test_same_input_fusion_is_the_members_side_by_side():
    """concat_qvb8r: the fused dict restores to the members' weights stacked, bit for bit (oracle decoder, CPU)."""
    from qvb8_b200 import fuse
    _, a = _pack(48, 256, seed=41, K=2, T=4)
    _, b = _pack(80, 256, seed=42, K=3, T=2)
    _, c = _pack(16, 256, seed=43, K=2, T=8)
    fused, splits = fuse.concat_qvb8r([a, b, c])
    assert splits == [48, 128] and fused["Q"] == 144 and fused["K"] == 7
    want = np.vstack([_dense(a), _dense(b), _dense(c)])
    assert np.array_equal(_dense(fused).view(np.uint32), want.view(np.uint32))
    blob = packs.write_qvb8r(fused, Q=fused["Q"], P=fused["P"], min_s=fused["min_s"], tau_s=fused["tau_s"],
                             esc_idx=fused["esc_idx"], esc_val=fused["esc_val"], esc_delta=fused["esc_delta"],
                             cert=dict(tau=fused["tau"], max_err=fused["max_err"]))
    assert np.array_equal(_dense(packs.read_qvb8r(blob)).view(np.uint32), want.view(np.uint32))


def test_tile_shards_are_the_rows_of_the_whole():
    """runs of whole tiles as tensors of their own (no re-encoding): restored, they are the whole tensor's rows; the
    escapes go with their rows; the bounds balance the coded words"""
    from qvb8_b200 import fuse
    _, d = _pack(200, 256, seed=61, K=3, T=4)
    whole = _dense(d)
    for world in (1, 2, 3, 8, 64):
        bounds = fuse.qvb8r_shard_bounds(d, world)
        assert bounds[0] == 0 and bounds[-1] == len(d["tiles"]) and all(a <= b for a, b in zip(bounds, bounds[1:]))
        got, seen, n_esc = np.zeros_like(whole), np.zeros(200, int), 0
        for r in range(world):
            sh, rows = fuse.qvb8r_tile_shard(d, bounds[r], bounds[r + 1])
            assert sh["Q"] == len(rows) and sh["words"].size == int(d["tile_off"][bounds[r + 1]] - d["tile_off"][bounds[r]])
            if sh["Q"]:
                got[rows] = _dense(sh)
            seen[rows] += 1
            n_esc += len(sh["esc_idx"])
            assert np.all(np.diff(sh["esc_idx"]) > 0)
        assert np.array_equal(got.view(np.uint32), whole.view(np.uint32)) and seen.min() == seen.max() == 1
        assert n_esc == len(d["esc_idx"])
        if world in (2, 3):
            sizes = [int(d["tile_off"][b] - d["tile_off"][a]) for a, b in zip(bounds, bounds[1:])]
            assert max(sizes) - min(sizes) <= 2 * int(np.diff(d["tile_off"]).max())
    with pytest.raises(ValueError):
        fuse.qvb8r_tile_shard(d, 3, len(d["tiles"]) + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 9, 40])
def test_tile_sharded_modules_cover_the_whole_product(cuda_lib, M):
    """three shard modules on one device, each with its run of tiles: their local rows, put in place, are the whole
    module's output"""
    from qvb8_b200.linear_r import QVBandLinearV8R, QVBandLinearV8RShard
    P = 512
    _, d = _pack(330, P, seed=71, K=3, T=4)
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.bfloat16)
    want = QVBandLinearV8R(d, device=DEV)(X).float()
    got = torch.full_like(want, float("nan"))
    for r in range(3):
        sh = QVBandLinearV8RShard(d, r, 3, device=DEV)
        got[:, sh.rows] = sh(X).float()
    assert torch.equal(got, want)
    one = QVBandLinearV8RShard(d, 0, 1, device=DEV)
    assert torch.equal(one(X).float(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 6, 14, 70])
def test_same_input_fusion_module(cuda_lib, M):
    """One module over the fused dict gives the members' module outputs side by side."""
    from qvb8_b200 import fuse
    from qvb8_b200.linear_r import QVBandLinearV8R
    P = 512
    ds = [_pack(Q, P, seed=50 + i, K=2, T=2)[1] for i, Q in enumerate((64, 32, 96))]
    fused, splits = fuse.concat_qvb8r(ds)
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.bfloat16)
    y = QVBandLinearV8R(fused, device=DEV)(X).float()
    parts = [QVBandLinearV8R(d, device=DEV)(X).float() for d in ds]
    got = torch.tensor_split(y, splits, dim=-1)
    for g, w in zip(got, parts):
        if M <= 16:
            assert torch.equal(g, w)                     # the same kernels on the same bytes
        else:
            assert torch.allclose(g, w, rtol=2e-2, atol=2e-2)        # library GEMM: the tile shape may differ


def _wide_symbols(Q, P, seed, K, T):
    """A coded tensor whose symbols reach beyond 512 (the factored product's limit)."""
    rng = np.random.default_rng(seed)
    d = rans.encode_ids(rng.integers(0, 1200, size=(Q, P)), K=K, T=T)
    tau_s = rng.uniform(1e-4, 2e-4, Q).astype(np.float32)
    d.update(Q=Q, P=P, min_s=(-600 * tau_s).astype(np.float32), tau_s=tau_s, esc_idx=np.zeros(0, np.int64),
             esc_val=np.zeros(0, np.float32), esc_delta=np.zeros(0, np.float32))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("Q,P,K,T,M,wide", [
    (1, 64, 1, 1, 2, False), (5, 192, 1, 2, 8, False), (37, 256, 2, 3, 5, False), (64, 320, 3, 8, 9, False),
    (130, 1088, 2, 5, 16, False), (90, 640, 2, 40, 7, False), (33, 512, 2, 4, 1, False), (40, 384, 1, 3, 6, True),
    (40, 384, 1, 3, 13, True)])
def test_gpu_products_at_tile_edges(cuda_lib, Q, P, K, T, M, wide):
    """Products where chunks (256 columns), pairs, four-tile CTAs, 32-row metadata groups and token fragments end early,
    and where the tensor-core form does not apply (large symbols, unaligned X).  fp32 sums of P terms: within TIGHT."""
    from qvb8_b200.ext_qvb8r import core_tensors, ext
    d = _wide_symbols(Q, P, Q + P, K, T) if wide else _pack(Q, P, seed=Q + P, K=K, T=T)[1]
    core = core_tensors(d, DEV)
    ids = oracle.rans_decode_ids(np.concatenate([d["words"], np.zeros(rans.PAD_WORDS, np.uint32)]),
                                 d["tile_off"].astype(np.int64), d["states"], d["tiles"].astype(np.int64),
                                 rans.slot_tables(d["freq"]), d["perm"], d["drow"].astype(np.int32), Q, P)
    band = oracle.rans_restore_f32(ids, d["min_s"], d["tau_s"])
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.float32)

    def check(x, rounded):
        W = band.astype(np.float16).astype(np.float32) if rounded else band
        want = x.double().cpu().numpy() @ W.astype(np.float64).T
        aligned = ext._mm(x, core, int(rounded))
        shifted = torch.empty(x.numel() + 1, dtype=x.dtype, device=DEV)[1:].view(x.shape).copy_(x)
        for got in (aligned, ext._mm(shifted, core, int(rounded))):
            assert np.linalg.norm(got.cpu().numpy() - want) <= TIGHT * np.linalg.norm(want)
        assert torch.equal(aligned, ext._mm(x, core, int(rounded)))
    check(X.half(), True)
    if M <= 8:
        check(X, False)
        check(X.bfloat16(), False)
        big = X.clone()
        big[M - 1] *= 1e36                                     # near the end of fp32's range
        check(big, False)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gpu_products_with_infinite_activations(cuda_lib, dtype):
    """an infinity times a finite weight is an infinity of the product's sign, a NaN stays with its token"""
    from qvb8_b200.ext_qvb8r import core_tensors, ext
    Q, P, M = 70, 384, 4
    _, d = _pack(Q, P, seed=3, K=2, T=3)
    core = core_tensors(d, DEV)
    X = synth.synth_activation(M, P, seed=1, device=DEV, dtype=torch.float32).to(dtype)
    clean = ext.multi(X, *core)
    X[1, 17], X[2, 300] = float("inf"), float("nan")
    got = ext.multi(X, *core)
    band = ext.decode(*core, P, 2, 0, core[4].numel() // 3, -1, 0)
    assert torch.equal(got[1], torch.where(band[:, 17] > 0, torch.inf, -torch.inf))
    assert torch.isnan(got[2]).all()
    tol = 1e-5 * clean.norm()                                  # (other tokens: the same sums, in the lane-by-lane order)
    assert (got[0] - clean[0]).norm() < tol and (got[3] - clean[3]).norm() < tol


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 17, 18, 32, 33, 48])
def test_linear_module_rows_and_types(cuda_lib, M, dtype):
    """every few-rows route of the module, with and without a bias, contiguous and not: product, escapes and narrowing"""
    from qvb8_b200.linear_r import QVBandLinearV8R
    Q, P = 150, 384
    _, d = _pack(Q, P, seed=31, K=3, T=3)
    assert len(d["esc_idx"]) > 0
    X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=dtype)
    want = X.double().cpu().numpy() @ _dense(d).astype(np.float64).T
    bias = torch.linspace(-1, 1, Q)
    strided = torch.empty(M, 2 * P, dtype=dtype, device=DEV)[:, ::2].copy_(X)
    tol = {torch.bfloat16: 4e-3, torch.float16: 1e-3, torch.float32: TIGHT if M <= 8 else 1e-3}[dtype]   # (from 9 rows on fp16 weights)
    for b in (None, bias):
        mod = QVBandLinearV8R(d, bias=b, device=DEV)
        ref = want if b is None else want + b.numpy()[None, :]
        y = mod(X)
        assert y.dtype == dtype and y.shape == (M, Q)
        assert np.linalg.norm(y.double().cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
        assert torch.equal(mod(strided), y)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [2, 17, 31, 33, 48])
def test_gpu_tc_rows_is_tc_for_more_rows(cuda_lib, M):
    from qvb8_b200.ext_qvb8r import Core, core_tensors, ext
    _, d = _pack(70, 704, seed=8, K=2, T=5)
    core = core_tensors(d, DEV)
    X = synth.synth_activation(M, 704, seed=M, device=DEV, dtype=torch.float16)
    got = ext.tc_rows(X, Core(704, core))
    want = torch.cat([ext._mm(x.contiguous(), core, 1) for x in X.split(16)]) if M % 16 != 1 else \
        torch.cat([ext._mm(x.contiguous(), core, 1) for x in X.split(15)])
    assert float((got - want).norm()) <= 1e-6 * float(want.norm())
    with pytest.raises(RuntimeError):
        ext.tc_rows(torch.zeros(49, 704, dtype=torch.float16, device=DEV), Core(704, core))


def test_the_kept_core_follows_its_tensors(monkeypatch):
    """the checked struct is rebuilt when a core tensor is replaced or its storage changes under it, and only then"""
    from qvb8_b200 import linear_r
    monkeypatch.setattr(linear_r, "Core", lambda P, core: type("Core", (), dict(core=core))())     # (the checks want a device)
    mod = linear_r.QVBandLinearV8R(_pack(40, 128, seed=2, K=1, T=2)[1], device="cpu")
    first = mod._core()[0]
    assert mod._core()[0] is first

    def swap_data():
        mod.words.data = mod.words.clone()

    def swap_storage():
        other = mod.tab.clone()
        mod.tab.set_(other.untyped_storage(), 0, other.shape)

    def swap_buffer():
        mod.tau_s = mod.tau_s.clone()
    for change in (swap_data, swap_storage, swap_buffer):
        change()
        again = mod._core()[0]
        assert again is not first and all(a is b for a, b in zip(again.core, mod.core()))
        assert mod._core()[0] is again
        first = again


def test_modules_saved_before_the_table_of_escape_rows():
    import copy
    import pickle

    from qvb8_b200.linear_r import QVBandLinearV8R
    mod = QVBandLinearV8R(_pack(40, 128, seed=2, K=1, T=2)[1], device="cpu")
    flat = mod.esc_flat.numpy()
    assert mod.esc_row.dtype == torch.int32 and np.array_equal(mod.esc_row.numpy(), np.searchsorted(flat, np.arange(41) * 128)) and flat.size
    old = copy.deepcopy(mod)
    del old._buffers["esc_row"]
    assert torch.equal(pickle.loads(pickle.dumps(old)).esc_row, mod.esc_row)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 12, 17, 48, 64])
@pytest.mark.parametrize("dtype", [torch.float64, torch.int32])
def test_linear_module_takes_other_types(cuda_lib, M, dtype):
    """activations that no kernel reads are computed as fp32 and the result comes back in their type, with and without a bias"""
    from qvb8_b200.linear_r import QVBandLinearV8R
    _, d = _pack(150, 384, seed=31, K=3, T=3)
    X = (3 * synth.synth_activation(M, 384, seed=M, device=DEV, dtype=torch.float32)).to(dtype)
    for b in (None, torch.linspace(-1, 1, 150)):
        mod = QVBandLinearV8R(d, bias=b, device=DEV)
        y = mod(X)
        assert y.dtype == dtype and torch.equal(y, mod(X.float()).to(dtype))


def _band64(d):
    ids = oracle.rans_decode_ids(np.concatenate([d["words"], np.zeros(rans.PAD_WORDS, np.uint32)]), d["tile_off"].astype(np.int64),
                                 d["states"], d["tiles"].astype(np.int64), rans.slot_tables(d["freq"]), d["perm"],
                                 d["drow"].astype(np.int32), int(d["Q"]), int(d["P"]))
    return oracle.rans_restore_f32(ids, d["min_s"], d["tau_s"])


@pytest.mark.gpu
@pytest.mark.parametrize("P", [640, 5120, 17408])
def test_gpu_tc_sums_against_64_bits(cuda_lib, P):
    """9 to 48 rows: products of fp16 numbers, summed two MMAs at a time and then in rounding fp32 additions.  Lane-by-lane sums,
    which these rows had before, are 9e-8 to 4e-7 away at these sizes; chains of MMAs as long as the row 2e-7 to 5e-6."""
    from qvb8_b200.ext_qvb8r import Core, core_tensors, ext
    _, d = _pack(60, P, seed=P, K=2, T=2)
    core = Core(P, core_tensors(d, DEV))
    W = torch.from_numpy(_band64(d)).to(DEV).half().double()
    for M in (9, 16, 32, 48):
        X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.float16)
        want = X.double() @ W.t()
        assert float((ext.tc_rows(X, core).double() - want).norm()) <= 3e-7 * float(want.norm()), M


@pytest.mark.gpu
@pytest.mark.parametrize("ids,middle", [((0, 8), 4), ((0, 41), 20), ((0, 41), 1500), ((0, 90), 256), ((900, 1300), 1100), ((0, 1200), 600)])
def test_gpu_factored_sums_against_64_bits(cuda_lib, monkeypatch, ids, middle):
    """2 to 8 rows of activations with a mean, over symbols that lie anywhere: the factored product counts from the row's zero
    weight and is as exact as fp32 sums of band values (4e-7 at 5120 columns), whatever the symbols (the coder puts a row's
    median id at symbol `middle`; readers take any)"""
    from qvb8_b200.ext_qvb8r import core_tensors, ext
    Q, P = 60, 5120
    monkeypatch.setattr(rans, "CENTRE", middle)
    rng = np.random.default_rng(ids[1])
    d = rans.encode_ids(rng.integers(*ids, size=(Q, P)), K=1, T=2)
    tau_s = rng.uniform(1e-3, 2e-3, Q).astype(np.float32)
    d.update(Q=Q, P=P, min_s=(-rng.uniform(*ids, size=Q) * tau_s).astype(np.float32), tau_s=tau_s, esc_idx=np.zeros(0, np.int64),
             esc_val=np.zeros(0, np.float32), esc_delta=np.zeros(0, np.float32))
    core = core_tensors(d, DEV)
    W = torch.from_numpy(_band64(d)).to(DEV).double()
    for M in (2, 5, 8):
        X = (synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.float32) + 1).bfloat16()
        want = X.double() @ W.t()
        for x in (X, X.float()):
            assert float((ext.multi(x, *core).double() - want).norm()) <= 4e-7 * float(want.norm()), (M, x.dtype)
