"""The work a user of this package has it do, as measurable cases: one pass = one call of the public entry points.

``listed()`` are the cases themselves, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` makes on the
GPU what a program holds before the call, ``run(state)`` is one pass, ``work(case)`` what a pass cannot do without, and
``tolerance(case)`` how far another correct implementation at the same precision may be off.

Kinds of pass (``op``):

* ``train``      ``ssd_mamba2`` forward and all gradients: the scan of a training step
* ``prefill``    ``ssd_mamba2`` forward only, state in and state out: reading a prompt, or one slice of it
* ``operator``   ``fused_ssd_scan`` with initial state and both outputs' gradients: the operator as such
* ``block``      the two ``fused_ssd_scan`` calls of a trapezoidal block, the second one on the first one's cache
* ``gated``      ``ssd_mamba2_gated``: the scan and the block's output stage, forward and all gradients
* ``mamba3``     ``ssd_mamba3``: rotary state angles and the trapezoidal form, forward and all gradients
* ``segmented``  ``ssd_mamba2_segmented``: one very long sequence on one GPU, forward and all gradients
* ``around``     the operators around the scan (coefficients, rotation of B and C, gated norm), forward and gradients
"""
import importlib
import math

import torch

import dhammic_ai_b200 as ssd

_split = importlib.import_module("dhammic-ai_b200.distributed")

_DT_BIAS0 = math.log(math.expm1(0.02))


def _case(name, op, dtype, batch, seqlen, nheads, headdim, d_state, ngroups, chunk):
    case = {"op": op, "dtype": dtype, "batch": batch, "seqlen": seqlen, "nheads": nheads, "headdim": headdim,
            "d_state": d_state, "ngroups": ngroups, "chunk": chunk}
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # full precision, the size on which correctness is checked while a model is being brought up
        _case("train_fp32_small", "train", "fp32", 2, 512, 8, 64, 64, 1, 64),
        # the tiny models (8 to 16 state columns, a few heads) that the operator's own tests stand for
        _case("operator_fp32_tiny", "operator", "fp32", 2, 512, 8, 32, 8, 8, 128),
        # one short slice of a prompt with the state carried in and out: a call where latency and launches count
        _case("prefill_slice", "prefill", "bf16", 1, 512, 24, 64, 128, 1, 64),
        # one long prompt of a large layer, batch 1: few (batch, head) pairs, many tiles each
        _case("prefill_long", "prefill", "bf16", 1, 16384, 64, 64, 128, 8, 128),
        # a training step of a 130M-parameter model's layer
        _case("train_130M", "train", "bf16", 8, 2048, 24, 64, 128, 1, 64),
        # a training step of a 1.3B-parameter model's layer, the benchmark's workload
        _case("train_1p3B", "train", "bf16", 16, 4096, 64, 64, 128, 8, 128),
        # a batch cut to a length that is a multiple of the chunk and of nothing more, 64 state columns, odd counts
        _case("train_ragged", "train", "bf16", 4, 1984, 20, 64, 64, 5, 64),
        # the operator as a block calls it: B and C per head, two scans that share one decay
        _case("block_bf16", "block", "bf16", 4, 2048, 16, 64, 128, 16, 128),
        # the scan with the gated norm behind it
        _case("gated_1p3B", "gated", "bf16", 4, 4096, 64, 64, 128, 8, 128),
        # the variant with rotary angles and the trapezoidal rule, at the size of the benchmark's configuration
        _case("mamba3_1p3B", "mamba3", "bf16", 16, 4096, 64, 64, 128, 8, 128),
        # one sequence of 131,072 positions on one GPU
        _case("segmented_131k", "segmented", "bf16", 1, 131072, 64, 64, 128, 8, 128),
        # what stands around the scan in a block, one micro-batch
        _case("around_1p3B", "around", "bf16", 4, 4096, 64, 64, 128, 64, 128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["train", "train", "train_fp32", "train_ragged", "operator", "prefill", "prefill_ragged", "block",
                     "gated", "mamba3", "segmented", "around"])
    ngroups = rng.choice([1, 1, 2, 4, 8])
    nheads = ngroups * rng.randint(max(1, 4 // ngroups), max(2, 64 // ngroups))
    chunk = rng.choice([64, 128, 128, 256])

    def sized(op, dtype, h, p, n, g, l, pairs, t_lo, t_hi, unit=None):
        """A length between t_lo and t_hi (a multiple of `unit`, and of the chunk), and a batch, with at most `pairs`
        (position, head) pairs in all."""
        unit = max(l, unit or l)
        t_hi = max(unit, min(t_hi, pairs // h))
        T = max(1, _log_int(rng, min(max(t_lo, unit), t_hi), t_hi) // unit) * unit
        b = _log_int(rng, 1, max(1, min(16, pairs // (h * T))))
        return _case(None, op, dtype, b, T, h, p, n, g, l)

    if op == "train_fp32":
        g = rng.choice([1, 2])
        return sized("train", "fp32", g * rng.randint(2, 8), rng.choice([32, 64]), rng.choice([16, 64, 128]), g,
                     rng.choice([32, 64, 100]), 16384, 200, 2048)
    if op == "operator":
        h = rng.randint(3, 8)
        return sized("operator", "fp32", h, rng.choice([16, 24, 32, 64]), rng.choice([8, 12, 16]), h, rng.choice([64, 128]),
                     16384, 128, 2048)
    if op in ("train_ragged", "prefill_ragged"):
        # lengths that are multiples of the chunk only; chunks that need not divide 128
        g = rng.choice([1, 2, 4])
        h = g * rng.randint(max(1, 4 // g), 32 // g)
        return sized(op.split("_")[0], "bf16", h, 64, rng.choice([64, 128]), g, rng.choice([32, 64, 80, 96]), 80000, 300, 4096)
    if op == "prefill":
        return sized("prefill", "bf16", nheads, 64, 128, ngroups, chunk, 1 << 20, 256, 32768, 128)
    if op == "block":
        h = rng.randint(4, 32)
        return sized("block", "bf16", h, 64, 128, h, chunk, 1 << 18, 256, 4096, 128)
    if op == "segmented":
        # a power-of-two length, which splits into segments of whole chunks
        return _case(None, "segmented", "bf16", 1, 1 << rng.randint(14, 17), nheads, 64, 128, ngroups, rng.choice([64, 128, 256]))
    if op == "around":
        return sized("around", "bf16", nheads, 64, rng.choice([64, 128]), nheads, 128, 1 << 20, 256, 4096, 64)
    return sized(op, "bf16", nheads, 64, 128, ngroups, chunk, 1 << 20 if op == "mamba3" else 1 << 21, 256, 8192, 128)


def prepare(case, seed):
    b, T, h, p, n, g = (case[k] for k in ("batch", "seqlen", "nheads", "headdim", "d_state", "ngroups"))
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    store = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def rand(*shape):
        return torch.rand(*shape, generator=gen, device="cuda")

    def leaf(t):
        return t.to(store).requires_grad_(True)

    s = {"case": case}
    if case["op"] == "around":
        s["leaves"] = [leaf(0.5 * randn(b, T, h) + _DT_BIAS0), leaf(randn(b, T, h)), (0.1 * randn(h)).requires_grad_(True),
                       (rand(h) * math.log(16.0)).requires_grad_(True),
                       leaf(randn(b, T, h, n) / math.sqrt(n)), leaf(randn(b, T, h, n) / math.sqrt(n)),
                       (torch.pi * (2 * rand(b, T, h, n // 2) - 1)).requires_grad_(True),
                       leaf(randn(b, T, h * p)), leaf(randn(b, T, h * p)), (1.0 + 0.1 * randn(h * p)).requires_grad_(True)]
        s["grads"] = ([randn(b, T, h).to(store) for _ in range(4)] + [randn(b, T, h, n).to(store) for _ in range(2)]
                      + [randn(b, T, h * p).to(store)])
        return s
    x, dy = randn(b, T, h, p), randn(b, T, h, p).to(store)
    dt = torch.nn.functional.softplus(0.5 * randn(b, T, h) + _DT_BIAS0).clamp_(1e-3, 1e-1)
    A_head = -torch.exp(rand(h) * math.log(16.0))
    B, C, D = randn(b, T, g, n) / math.sqrt(n), randn(b, T, g, n) / math.sqrt(n), randn(h)
    if case["op"] == "operator":
        init = 0.5 * randn(b, 1, h, p, n)
        s["leaves"] = [leaf(x * dt.unsqueeze(-1)), leaf(dt * A_head), leaf(B), leaf(C), leaf(init)]
        s["grads"] = [dy, randn(b, h, p, n).to(store)]
    elif case["op"] == "block":
        lam = torch.sigmoid(randn(b, T, h))
        a = dt * A_head
        gamma, beta = lam * dt, (1.0 - lam) * dt * torch.exp(a)
        pad = torch.nn.functional.pad
        s["leaves"] = [leaf(x * gamma.unsqueeze(-1)), leaf(a), leaf(B), leaf(C),
                       leaf(pad(x[:, :-1], (0, 0, 0, 0, 1, 0)) * beta.unsqueeze(-1)), leaf(pad(B[:, :-1], (0, 0, 0, 0, 1, 0)))]
        s["grads"] = [dy, dy]
    elif case["op"] == "prefill":
        s["inputs"] = [x.to(store), dt, A_head, B.to(store), C.to(store), D]
        s["init"] = 0.5 * randn(b, h, p, n)
    else:
        s["leaves"] = [leaf(x), dt.requires_grad_(True), A_head.requires_grad_(True), leaf(B), leaf(C), D.requires_grad_(True)]
        s["grads"] = [dy]
        if case["op"] == "gated":
            s["leaves"] += [leaf(randn(b, T, h * p)), (1.0 + 0.1 * randn(h * p)).requires_grad_(True)]
        elif case["op"] == "mamba3":
            s["leaves"] += [leaf(torch.pi * (2 * rand(b, T, h, n // 2) - 1) * torch.sigmoid(randn(b, T, h, n // 2))),
                            torch.sigmoid(randn(b, T, h)).requires_grad_(True)]
    return s


def run(s):
    case = s["case"]
    op, chunk = case["op"], case["chunk"]
    if op == "prefill":
        with torch.no_grad():
            return ssd.ssd_mamba2(*s["inputs"], chunk, s["init"])
    lv = s["leaves"]
    if op == "train":
        outs = [ssd.ssd_mamba2(*lv, chunk)[0]]
    elif op == "operator":
        outs = list(ssd.fused_ssd_scan(*lv[:4], chunk, lv[4])[:2])
    elif op == "block":
        y1, _, cache = ssd.fused_ssd_scan(*lv[:4], chunk)
        outs = [y1, ssd.fused_ssd_scan(lv[4], lv[1], lv[5], lv[3], chunk, None, cache)[0]]
    elif op == "gated":
        outs = [ssd.ssd_mamba2_gated(*lv, 1e-6, chunk)[0]]
    elif op == "mamba3":
        outs = [ssd.ssd_mamba3(*lv, chunk)]
    elif op == "segmented":
        outs = [_split.ssd_mamba2_segmented(*lv, chunk)[0]]
    else:
        dt_raw, lam_raw, dt_bias, A_log, B, C, angles, y, z, weight = lv
        outs = list(ssd.fused_trapezoidal(dt_raw, lam_raw, dt_bias, A_log))
        outs += [ssd.fused_rope(B, angles), ssd.fused_rope(C, angles), ssd.fused_gate_norm(y, z, weight, 1e-6)]
    return [o.detach() for o in outs] + list(torch.autograd.grad(outs, lv, s["grads"]))


def work(case):
    """Bytes: every input read once and every output written once per direction (the backward reads its inputs again).
    Operations: the products of the chunked form on tiles of at most 128 positions, C B^T once per group (per head for the
    rotated form), forward, and twice that for the backward."""
    b, T, h, p, n, g = (case[k] for k in ("batch", "seqlen", "nheads", "headdim", "d_state", "ngroups"))
    op, l = case["op"], min(case["chunk"], 128)
    w = 2 if case["dtype"] == "bf16" else 4
    tok, ex, eb, state = b * T, h * p, g * n, 4 * b * h * p * n
    gcb = h if op == "mamba3" else g
    fwd = tok * (2 * l * gcb * n + h * (2 * l * p + 4 * n * p))
    all_ = fwd + tok * (6 * l * gcb * n + h * (4 * l * p + 8 * n * p))
    if op == "around":
        rope = 2 * tok * h * (5 * n * w + 3 * (n // 2) * 4)
        return {"bytes": rope + 14 * tok * h * w + 8 * tok * ex * w, "flops": tok * h * (60 * n + 40 + 40 * p)}
    if op == "prefill":
        return {"bytes": tok * (2 * ex * w + 2 * eb * w + 4 * h) + 2 * state, "flops": fwd}
    if op == "operator":
        return {"bytes": tok * w * (5 * ex + 6 * eb + 3 * h) + 5 * state // 4 * w, "flops": all_}
    if op == "block":  # two scans: x, y, dy, dx and B, dB each; a, C, da, dC shared (read again by the backward)
        return {"bytes": tok * w * (10 * ex + 6 * eb + 3 * eb + 3 * h), "flops": 2 * all_}
    step = tok * (5 * ex * w + 6 * eb * w + 12 * h)
    if op == "gated":  # z in, out out; z, y, dout in and dz, dy out again
        step += tok * ex * w * 5
    if op == "mamba3":
        step += tok * h * (3 * w * (n // 2) + 12)
    return {"bytes": step, "flops": all_}


def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}  # sums of a few hundred to a few thousand fp32 terms, some of which cancel (decay gradients)
    if case["op"] == "mamba3":
        return {"rel": 2e-2}  # the angle gradient is a running sum along the sequence of bf16-rounded terms
    return {"rel": 1e-2}
