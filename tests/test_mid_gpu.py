"""The tcgen05 kernel for a dozen to a few hundred tokens against the oracle's dense fp32 product on the restored weights."""
import numpy as np
import pytest
import torch

import oracle
from qvb8_b200 import lib, synth
from util import pack_np, random_pack, rel_fro

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TIGHT = 1e-6        # exact products, sums of at most 24 truncating and then rounding fp32 additions (measured: 2e-7)


def _operands(pk):
    st, keep = lib.pack_struct(pk.ids, pk.min_s, pk.tau_s, pk.nbits, pk.bit_off, pk.P, pk.esc_idx, pk.esc_vals)
    return st, keep, lib.build_plan(st, keep)


@pytest.mark.parametrize("Q,P,M,widths,esc", [
    (128, 64, 9, (7,), 0.0),                       # one K block: an odd last pair, one run
    (1, 128, 16, (6,), 0.0),                       # one row
    (256, 512, 17, (6, 7, 8), 0.0),                # token tiles of 32
    (200, 1024, 33, (3, 5, 7, 8), 0.002),          # 64; ragged rows, escapes
    (384, 256, 70, (4, 9, 12), 0.001),             # 96; 12-bit rows are recomputed in fp32, with escapes on top
    (300, 1280, 128, (1, 2, 10, 11, 14), 0.0),     # every unpack mode
    (130, 320, 129, (3, 6, 7, 8), 0.001),          # two token tiles; five K blocks
    (64, 192, 16, (5, 7), 0.0),                    # rows that do not start on 16 bytes take the id-by-id path
    (2500, 2048, 24, (7, 8), 0.001),               # runs that cut tiles at every place: 21 row tiles over 80 runs
    (6000, 4096, 40, (6, 7), 0.001),               # 148 runs
    (16500, 384, 48, (7,), 0.0),                   # whole tiles, one per run
])
def test_mid_matches_oracle(cuda_lib, Q, P, M, widths, esc):
    pk = random_pack(Q, P, widths, seed=Q + M, esc_frac=esc, device=DEV)
    st, keep, plan = _operands(pk)
    dense = oracle.qvb8_dense(pack_np(pk))
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        X = synth.synth_activation(M, P, seed=M, device=DEV, dtype=dt)
        Y = lib.mid_m(st, keep, X, plan)
        want = oracle.matmul_f32w(X.float().cpu().numpy(), dense, narrow_x=True)
        err = rel_fro(Y.cpu().numpy(), want)
        assert err < TIGHT, (dt, err)
        assert torch.equal(Y, lib.mid_m(st, keep, X, plan))            # the runs' parts are added in one order
    assert lib.device_status() == 0


def test_mid_keeps_the_activations_range_in_mode_1(cuda_lib):
    """x_mode 1: activations beyond fp16's range are prescaled per token by a power of two, results scaled back"""
    Q, P, M = 300, 512, 20
    pk = random_pack(Q, P, (6, 7, 12), seed=5, esc_frac=0.002, device=DEV)
    st, keep, plan = _operands(pk)
    X = synth.synth_activation(M, P, seed=3, device=DEV, dtype=torch.float32)
    X[3] *= 3e6
    X[7] *= 1e30
    X = X.to(torch.bfloat16)
    Y = lib.mid_m(st, keep, X, plan, x_mode=1).double().cpu().numpy()
    want = X.double().cpu().numpy() @ oracle.qvb8_dense(pack_np(pk)).astype(np.float64).T
    for m in range(M):                                                  # per token: the magnitudes differ by 30 decades
        assert np.linalg.norm(Y[m] - want[m]) < 1e-3 * np.linalg.norm(want[m]), m   # (fp16 subnormals of scaled tokens)
    assert lib.device_status() == 0


@pytest.mark.parametrize("M", [9, 16, 50, 96])
def test_calls_that_take_the_mid_route_agree_with_the_streaming_kernel(cuda_lib, M):
    """The dispatch by rows, scratch and alignment: qvb8_small_m_ex with its full scratch and with no more than the
    streaming kernel needs, unaligned and strided activations, the module and the extension's forward."""
    import ctypes
    from qvb8_b200.ext_qvb8 import ext
    from qvb8_b200.linear import QVBandLinearV8
    Q, P = 300, 512
    pk = synth.synth_pack(Q, P, seed=3, tau=2e-3, device=DEV, restore="fp16+bf16")
    st, keep, plan = _operands(pk)
    X = synth.synth_activation(M, P, seed=M, device=DEV)
    want = oracle.matmul_f32w(X.float().cpu().numpy(), oracle.qvb8_dense(pack_np(pk)), narrow_x=True)
    args = (pk.ids, pk.min_s, pk.nbits, pk.bit_off, P, pk.tau_s, pk.esc_idx, pk.esc_vals)
    shifted = torch.empty(X.numel() + 1, dtype=X.dtype, device=DEV)[1:].view(M, P).copy_(X)
    strided = torch.empty(M, 2 * P, dtype=X.dtype, device=DEV)[:, ::2].copy_(X)
    got = [ext.forward(x, *args) for x in (X, shifted, strided)]
    if M <= 48:
        got.append(lib.small_m(st, keep, X, plan=plan))
        L, Y = lib.load(), torch.empty(M, Q, device=DEV)
        small = torch.zeros(1 << 18, dtype=torch.uint8, device=DEV)     # the counters alone: the streaming kernel's scratch
        lib.check(L.qvb8_small_m_ex(ctypes.byref(st), plan.data_ptr(), X.data_ptr(), lib.dtype_code(X.dtype), 0, M, Y.data_ptr(),
                                    small.data_ptr(), small.numel(), 0, lib.stream_ptr(X.device)), "small_m_ex")
        got.append(Y)
        full = lib.scratch_for(X.device, int(L.qvb8_small_m_scratch_bytes(M, Q, P)))
        assert int(full[:1 << 18].count_nonzero()) == 0                 # the streaming kernel's counters stay zero
    for y in got:
        assert rel_fro(y.cpu().numpy(), want) < 1e-3                    # (a dense fp16 copy for the unaligned 50 and 96 rows)
    lin = QVBandLinearV8.from_pack(pk)
    wantb = oracle.matmul_f32w(X.float().cpu().numpy(), oracle.qvb8_dense(pack_np(pk), table="bf16"), narrow_x=False)
    for x in (X, shifted, strided):
        assert rel_fro(lin(x).float().cpu().numpy(), wantb) < 1e-2      # bf16 results
    assert rel_fro(lin(X.float()).cpu().numpy(), want) < TIGHT
    assert lib.device_status() == 0


@pytest.mark.parametrize("P", [4096, 12288, 17408])
def test_mid_sums_against_64_bits(cuda_lib, P):
    """fp32 results of activations that fp16 holds exactly, without and with a mean: the streaming kernel, which takes these
    rows in lists, is 6e-7 to 1.6e-6 away at these sizes, and up to 2e-4 with a mean.  Here chunks of 384 columns (24 additions
    that truncate, 2^-24 of the chunk's sum each) are added with rounding: under 5e-7, and 1e-6 where sums of 17408 activations
    with a mean meet a rest of half a step."""
    import ctypes
    pk = synth.synth_pack(300, P, seed=P, device=DEV)
    st, keep, plan = _operands(pk)
    W = torch.from_numpy(oracle.qvb8_dense(pack_np(pk))).to(DEV).double()
    L = lib.load()
    for M in (9, 16, 48, 96):
        for mean, bound in ((0.0, 5e-7), (1.0, 1e-6)):
            X = (synth.synth_activation(M, P, seed=M, device=DEV, dtype=torch.float32) + mean).half().float()
            want = X.double() @ W.t()
            away = lambda Y: float((Y.double() - want).norm() / want.norm())
            err = away(lib.mid_m(st, keep, X, plan))
            assert err < bound, (M, mean, err)
            if M <= 48:                                                 # the streaming kernel: a scratch too small for the other
                less = (1 << 18) + int(L.qvb8_mid_m_scratch_bytes(M, 300, P)) - 1
                small, Y = torch.zeros(less, dtype=torch.uint8, device=DEV), torch.empty(M, 300, device=DEV)
                lib.check(L.qvb8_small_m_ex(ctypes.byref(st), plan.data_ptr(), X.data_ptr(), lib.dtype_code(X.dtype), 0, M, Y.data_ptr(),
                                            small.data_ptr(), less, 0, lib.stream_ptr(X.device)), "small_m_ex")
                assert err <= away(Y), (M, mean)


def test_mid_in_a_graph(cuda_lib):
    """captured with its three launches and replayed on new activations"""
    pk = synth.synth_pack(700, 2048, seed=4, device=DEV)
    st, keep, plan = _operands(pk)
    X = synth.synth_activation(20, 2048, seed=1, device=DEV)
    lib.mid_m(st, keep, X, plan)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        Y = lib.mid_m(st, keep, X, plan)
    X.copy_(synth.synth_activation(20, 2048, seed=2, device=DEV))
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(Y, lib.mid_m(st, keep, X, plan))
