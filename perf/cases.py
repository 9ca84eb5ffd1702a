"""The work this package is timed on: packed linears, the decode stack, the expert layer and entropy-coded linears.

Sizes are those of the benchmark configurations (9B-, 27B-class dense decoders, 35B-A3B-class expert layer); weights are
N(0, 0.02) with 0.1 % outliers, activations N(0, 1), as those configurations state.  `listed` holds the cases, `draw` one
more of the same ranges, `prepare` / `run` the state a user's program keeps and one pass through the public modules,
`exact` the same result in 64 bits from the packs' bytes with plain torch.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from qvb8_b200 import experts, fuse, stack, synth
from qvb8_b200.linear import QVBandLinearV8
from qvb8_b200.linear_r import QVBandLinearV8R

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DEV = "cuda:0"


def listed():
    def linear(name, Q, P, M, dtype="bf16", certified=False, tau=1e-3):
        return dict(name=name, kind="linear", Q=Q, P=P, M=M, dtype=dtype, certified=certified, tau=tau)

    def coded(name, Q, P, M, copies, dtype="bf16"):
        return dict(name=name, kind="coded", Q=Q, P=P, M=M, copies=copies, dtype=dtype)

    def moe(name, M):
        return dict(name=name, kind="moe", M=M, experts=128, topk=8, d=2048, f=768, act="silu", dtype="bf16")

    return [
        # one token through the narrowest projection of a 9B-class layer: the smallest call, launch and host time count
        linear("linear-k-9b-m1", 1024, 4096, 1),
        # speculative verification of 8 draft tokens, 9B-class down projection (long rows)
        linear("linear-down-9b-m8", 4096, 12288, 8),
        # verification of 13 tokens (an odd draft length) in fp16, 27B-class gate projection
        linear("linear-gate-27b-m13", 17408, 5120, 13, dtype="fp16", tau=2e-3),
        # a short prompt, 9B-class o projection, pack certified for bf16
        linear("linear-o-9b-m300", 4096, 4096, 300, certified=True),
        # a prefill chunk through the 27B-class gate projection: the largest call
        linear("linear-gate-27b-m2048", 17408, 5120, 2048, tau=2e-3),
        # one decode step of a 9B-class linear stack (8 of its layers behind one launch), replayed as a graph
        dict(name="stack-9b-m1", kind="stack", config="9b-dense", layers=8, M=1),
        # the same stack verifying 8 tokens
        dict(name="stack-9b-m8", kind="stack", config="9b-dense", layers=8, M=8),
        # the 35B-A3B-class expert layer for 8 tokens (decode of a few sequences) and for 32 (a batch, or a verify step)
        moe("moe-35b-m8", 8),
        moe("moe-35b-m32", 32),
        # entropy-coded packs, 27B-class: one token through q, 12 verify tokens through gate, a prompt through down
        coded("coded-q-27b-m1", 5120, 5120, 1, 4),
        coded("coded-gate-27b-m12", 17408, 5120, 12, 8),
        coded("coded-down-27b-m512", 5120, 17408, 512, 8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["stack"] + ["moe"] * 2 + ["coded"] * 3)
    if kind == "linear":
        lo, hi = rng.choice([(1, 1), (2, 8), (9, 48), (49, 96), (97, 2048)])
        Q, P, M = _log(rng, 700, 24576), 128 * _log(rng, 8, 96), _log(rng, lo, hi)
        while Q * P * M > 17408 * 5120 * 2048:
            M //= 2
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        return dict(kind=kind, Q=Q, P=P, M=M, dtype=dtype, certified=dtype == "bf16" and rng.random() < 0.4,
                    tau=rng.choice([1e-3, 2e-3]))
    if kind == "stack":
        return dict(kind=kind, config="9b-dense", layers=rng.randint(1, 8), M=_log(rng, 1, 16))
    if kind == "moe":
        E = rng.choice([32, 64, 128])
        return dict(kind=kind, M=_log(rng, 1, 48), experts=E, topk=rng.randint(2, 8), d=128 * rng.randint(8, 24),
                    f=128 * rng.randint(3, 10), act=rng.choice(["silu", "silu", "relu2"]),
                    dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]))
    lo, hi = rng.choice([(1, 1), (2, 8), (9, 16), (17, 48), (49, 512)])
    copies = rng.randint(1, 6)
    return dict(kind=kind, Q=copies * _log(rng, 300, 1400), P=128 * _log(rng, 8, 80), M=_log(rng, lo, hi), copies=copies,
                dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]))


# ---- inputs ---------------------------------------------------------------------------------------------------

def _activation(case, P, seed):
    return synth.synth_activation(case["M"], P, seed=seed + 7, device=DEV, dtype=DTYPES[case["dtype"]])


def _linear_pack(case, seed):
    return synth.synth_pack(case["Q"], case["P"], seed, tau=case["tau"], device=DEV,
                            restore="fp16+bf16" if case["certified"] else "fp16")


def _coded_pack(case, seed):
    """A `.qvb8r` tensor of Q rows: rows / copies are coded once and laid side by side (each copy's band scaled by its
    own power of two), because the coder is slow and the decoder's work does not depend on which rows repeat."""
    rows = case["Q"] // case["copies"]
    W = synth.synth_weight(rows, case["P"], seed, device=DEV)
    one = synth.encode_qvb8r(W, tau=2e-3, K=2, T=max(1, -(-case["Q"] // 4096)))
    members = []
    for k in range(case["copies"]):
        f = np.float32(2.0 ** -(k % 4))
        members.append({**one, **{n: np.asarray(one[n], np.float32) * f
                                  for n in ("min_s", "tau_s", "esc_val", "esc_delta")}})
    return fuse.concat_qvb8r(members)[0] if case["copies"] > 1 else one


def _expert_packs(case, seed):
    """One tall pack per projection, cut into the experts' packs."""
    E, d, f = case["experts"], case["d"], case["f"]
    up_rows = 2 * f if case["act"] == "silu" else f

    def cut(rows, cols, s):
        per = max(1, (1 << 26) // (rows * cols))
        out = []
        for e0 in range(0, E, per):
            n = min(per, E - e0)
            tall = synth.encode_qvb8(synth.synth_weight(n * rows, cols, s + e0, device=DEV), tau=1e-3, policy="inband")
            out += [fuse.row_shard(tall, i * rows, (i + 1) * rows) for i in range(n)]
        return out
    return cut(up_rows, d, seed), cut(d, f, seed + 500)


def _routing(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 11)
    logits = torch.randn(case["M"], case["experts"], generator=g, device=DEV)
    w, idx = torch.topk(torch.softmax(logits, dim=-1), case["topk"], dim=-1)
    return idx, w / w.sum(dim=-1, keepdim=True)


def _stack(case, seed):
    cfg = dataclasses.replace(stack.CONFIGS[case["config"]], layers=case["layers"])
    s = stack.LinearStack(cfg, case["M"], DEV, seed_base=seed)
    for i, x in enumerate(s.x.values()):
        x.copy_(synth.synth_activation(case["M"], x.shape[1], seed=seed + 7 + i, device=DEV))
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        return dict(layer=QVBandLinearV8.from_pack(_linear_pack(case, seed)), x=_activation(case, case["P"], seed))
    if kind == "coded":
        return dict(layer=QVBandLinearV8R(_coded_pack(case, seed), device=DEV), x=_activation(case, case["P"], seed))
    if kind == "moe":
        up, down = _expert_packs(case, seed)
        layer = experts.QVBandExpertsV8(up, down, num_experts=case["experts"], act=case["act"])
        idx, w = _routing(case, seed)
        return dict(layer=layer, x=_activation(case, case["d"], seed), idx=idx, w=w)
    s = _stack(case, seed)
    s.set_grouping(case["layers"])
    s.capture()
    return dict(stack=s)


def run(state):
    if "stack" in state:
        state["stack"].step()
        return [y for layer in state["stack"].y_launch for y in layer]
    if "idx" in state:
        return state["layer"](state["x"], state["idx"], state["w"])
    return state["layer"](state["x"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------

def _linear_bytes(Q, P, M, size, bits, escapes=1e-3):
    return Q * P * bits / 8 + 17 * Q + 12 * escapes * Q * P + M * (P + Q) * size


def work(case):
    kind, M = case["kind"], case["M"]
    size = 4 if case.get("dtype") == "fp32" else 2
    if kind == "linear":
        bits = 7 if case["tau"] == 1e-3 else 6
        return dict(bytes=_linear_bytes(case["Q"], case["P"], M, size, bits), flops=2 * case["Q"] * case["P"] * M)
    if kind == "coded":                                                  # the coder leaves 4.4 bits a weight at this tau
        return dict(bytes=_linear_bytes(case["Q"], case["P"], M, size, 4.4) + 256 * case["Q"] / max(1, -(-case["Q"] // 4096)),
                    flops=2 * case["Q"] * case["P"] * M)
    if kind == "moe":
        E, d, f, k = case["experts"], case["d"], case["f"], case["topk"]
        distinct = E * (1 - (1 - k / E) ** M)
        per = (3 if case["act"] == "silu" else 2) * d * f
        return dict(bytes=distinct * per + 2 * M * d * size, flops=2 * per * M * k)
    cfg = stack.CONFIGS[case["config"]]
    total = sum(_linear_bytes(q, p, M, 3, 7) for _, q, p, _ in cfg.projections())
    return dict(bytes=case["layers"] * total, flops=2 * case["layers"] * cfg.weights_per_layer() * M)


def tolerance(case):
    """About four times the measured distance from the 64-bit result: the rounding of the output (1.7e-3 in bf16, 2.1e-4 in
    fp16), the narrowing of activations or weights to fp16 that every route but the coded one up to 8 rows has (2.1e-4 to
    3.2e-4), and 32-bit sums where neither is seen (1.6e-6: bf16 activations are exact in fp16)."""
    if case["kind"] == "stack":
        return dict(rel=7e-6)
    if case["dtype"] == "bf16":
        return dict(rel=7e-3)
    if case["dtype"] == "fp32" and case["kind"] == "coded" and case["M"] <= 8:
        return dict(rel=7e-6)
    return dict(rel=1.3e-3)


# ---- the same results in 64 bits, from the packs' bytes, with plain torch ---------------------------------------

def _restore64(Q, P, ids, nbits, bit_off, min_s, tau_s, esc_idx=None, esc_vals=None):
    W = torch.empty(Q, P, dtype=torch.float64, device=DEV)
    nb = nbits.to(torch.int64)
    raw = torch.cat([ids, ids.new_zeros(8)])
    cols = torch.arange(P, device=DEV)
    step = max(1, (1 << 25) // P)
    for r in range(0, Q, step):
        n = nb[r:r + step, None]
        bit = bit_off[r:r + step, None] + cols * n
        byte = bit >> 3
        word = raw[byte].to(torch.int64) | (raw[byte + 1].to(torch.int64) << 8) | (raw[byte + 2].to(torch.int64) << 16)
        code = (word >> (bit & 7)) & ((1 << n) - 1)
        W[r:r + step] = code.double() * tau_s[r:r + step, None].double() + min_s[r:r + step, None].double()
    if esc_idx is not None and esc_idx.numel():
        W.view(-1)[esc_idx] = esc_vals.double()
    return W


def _restore_coded64(d):
    """rANS decoding, all tiles at once: 32 states a tile, symbols in pairs, then the states below 2^32 take a word."""
    Q, P = int(d["Q"]), int(d["P"])
    up = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).astype(dt)).to(DEV)
    freq = np.asarray(d["freq"], np.int64)
    slots = np.zeros((3, freq.shape[0], 4096), np.int64)
    for k, f in enumerate(freq):
        sym = np.repeat(np.arange(f.size), f)
        slots[:, k] = sym, np.arange(4096) - (np.cumsum(f) - f)[sym], f[sym]
    slots = up(slots.reshape(3, -1), np.int64)
    words = up(np.concatenate([np.asarray(d["words"], np.int64), np.zeros(64, np.int64)]), np.int64)
    tiles = up(np.asarray(d["tiles"]).reshape(-1, 3), np.int64)
    x = torch.from_numpy(np.ascontiguousarray(d["states"], np.uint64).reshape(-1, 32).view(np.int64)).to(DEV)
    cursor = up(np.asarray(d["tile_off"])[:-1], np.int64)
    codes = torch.zeros(Q, P, dtype=torch.int64, device=DEV)
    low = (1 << 52) - 1                                                   # a logical shift right by 12 of a signed word
    for r in range(int(tiles[:, 2].max())):
        live = torch.nonzero(tiles[:, 2] > r).view(-1)
        base = tiles[live, 0, None] * 4096
        xs, cur = x[live], cursor[live]
        row = torch.empty(live.numel(), P // 32, 32, dtype=torch.int64, device=DEV)
        for s in range(P // 32):
            slot = base + (xs & 4095)
            row[:, s] = slots[0][slot]
            xs = slots[2][slot] * ((xs >> 12) & low) + slots[1][slot]
            if s % 2:
                need = (xs >> 32) == 0
                rank = torch.cumsum(need, 1)
                xs = torch.where(need, (xs << 32) | words[cur[:, None] + rank - 1], xs)
                cur = cur + rank[:, -1]
        x[live], cursor[live] = xs, cur
        codes[tiles[live, 1] + r] = row.view(-1, P)
    perm = up(d["perm"], np.int64)
    W = torch.empty(Q, P, dtype=torch.float64, device=DEV)
    W[perm] = codes.double()
    W += up(d["drow"], np.float64)[:, None]
    W = W * up(d["tau_s"], np.float64)[:, None] + up(d["min_s"], np.float64)[:, None]
    if len(d["esc_idx"]):
        W.view(-1)[up(d["esc_idx"], np.int64)] = up(d["esc_val"], np.float64)
    return W


def _pack64(pk, table="fp16"):
    idx, vals = (pk.esc_idx_bf16, pk.esc_vals_bf16) if table == "bf16" else (pk.esc_idx, pk.esc_vals)
    return _restore64(pk.Q, pk.P, pk.ids, pk.nbits, pk.bit_off, pk.min_s, pk.tau_s, idx, vals)


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        x = _activation(case, case["P"], seed).double()
        return x @ _pack64(_linear_pack(case, seed), "bf16" if case["certified"] and 8 <= case["M"] <= 96 else "fp16").t()
    if kind == "coded":
        return _activation(case, case["P"], seed).double() @ _restore_coded64(_coded_pack(case, seed)).t()
    if kind == "stack":
        s = _stack(case, seed)
        return [s.x[xname].double() @ _pack64(pk).t() for layer in s.launches for _, pk, _, _, xname, _ in layer]
    ups, downs = _expert_packs(case, seed)
    idx, w = _routing(case, seed)
    x = _activation(case, case["d"], seed).double()
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        tok, j = torch.nonzero(idx == e, as_tuple=True)
        if not tok.numel():
            continue
        h = x[tok] @ _pack64(ups[e]).t()
        if case["act"] == "silu":
            gate, h = h.chunk(2, dim=1)
            h = gate * torch.sigmoid(gate) * h
        else:
            h = torch.relu(h) ** 2
        out.index_add_(0, tok, (h @ _pack64(downs[e]).t()) * w[tok, j, None].double())
    return out
