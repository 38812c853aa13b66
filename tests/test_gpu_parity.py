"""GPU parity tests: the CUDA path, called through the C ABI by the operator, against the CPU oracle
and the golden fixtures.  Metric: max|a-b| / max|b| per output tensor; bars: 1e-4 for fp32,
2e-2 for bf16 inputs with fp32 accumulation (the oracle then runs in fp32 on the bf16-rounded inputs,
as the reference's own bf16 test does, tests/kernels/test_ssd_scan.py:74-96)."""
import glob
from dataclasses import replace

import numpy as np
import pytest
import torch

from conftest import GOLDEN, TOL_BF16, TOL_FP32, load_golden, rel_err

pytestmark = pytest.mark.gpu

DEV = "cuda"
REF_CASES = sorted(p.split("/")[-1] for p in glob.glob(str(GOLDEN / "ref_*.npz")))


def _t(a, dtype=None):
    t = torch.from_numpy(np.asarray(a))
    return t if dtype is None else t.to(dtype)


def run_operator(pkg, x, A, B, C, chunk, init=None, dY=None, dfinal=None, cache=None):
    """fused_ssd_scan forward + backward on the GPU; returns CPU tensors."""
    leaves = [t.detach().to(DEV).requires_grad_(True) for t in (x, A, B, C)]
    il = init.detach().to(DEV).requires_grad_(True) if init is not None else None
    Y, fs, ch = pkg.fused_ssd_scan(*leaves, chunk, il, cache)
    res = {"Y": Y.detach().cpu(), "final": fs.detach().cpu(), "cache": ch}
    if dY is not None:
        outs, gouts = [Y], [dY.to(DEV).to(Y.dtype)]
        if dfinal is not None:
            outs.append(fs)
            gouts.append(dfinal.to(DEV).to(fs.dtype))
        ins = leaves + ([il] if il is not None else [])
        grads = torch.autograd.grad(outs, ins, gouts, allow_unused=True)
        for k, g in zip(("dx", "dA", "dB", "dC", "dinit"), grads):
            res[k] = None if g is None else g.detach().cpu()
    torch.cuda.synchronize()
    return res


@pytest.fixture
def tensor_cores(pkg):
    """The tensor-core kernels also for shapes that they are not chosen for."""
    pkg.set_kernel_path("tc")
    yield
    pkg.set_kernel_path("auto")


@pytest.mark.parametrize("name", REF_CASES)
def test_fp32_against_reference_fixtures(pkg, cabi, name):
    g = load_golden(name)
    chunk = int(g["chunk"])
    init = _t(g["init"]) if g["init"].size else None
    dfinal = _t(g["dfinal"]) if g["dfinal"].size else None
    r = run_operator(pkg, _t(g["x"]), _t(g["A"]), _t(g["B"]), _t(g["C"]), chunk, init, _t(g["dY"]), dfinal)
    assert rel_err(r["Y"], _t(g["Y"])) < TOL_FP32
    assert rel_err(r["final"], _t(g["final_state"])) < TOL_FP32
    assert rel_err(r["cache"]["A_cumsum"], _t(g["A_cumsum"])) < TOL_FP32
    for k in ("dx", "dA", "dB", "dC"):
        assert rel_err(r[k], _t(g[k])) < TOL_FP32, k
    if init is not None:
        assert rel_err(r["dinit"], _t(g["dinit"])) < TOL_FP32
    # cached second call (the caller's beta path): same A and C, shifted x and B; no decay gradient
    r2 = run_operator(pkg, _t(g["x2"]), _t(g["A"]), _t(g["B2"]), _t(g["C"]), chunk, None, _t(g["dY"]), None,
                      cache=r["cache"])
    assert rel_err(r2["Y"], _t(g["Y_cached"])) < TOL_FP32
    assert r2["dA"] is None
    for k in ("dx", "dB", "dC"):
        assert rel_err(r2[k], _t(g[k + "_cached"])) < TOL_FP32, k


@pytest.mark.parametrize("shape", [(2, 512, 4, 32, 8), (2, 256, 4, 16, 8), (1, 1024, 4, 16, 8), (2, 512, 8, 32, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_reference_test_shapes(pkg, cabi, oracle, shape, dtype):
    """Shapes, value ranges and chunk size of the reference's own scan tests
    (tests/kernels/test_ssd_scan.py:31-52), forward and gradients."""
    b, T, h, p, n = shape
    x, A, B, C = pkg.make_reference_test_inputs(b, T, h, p, n, dtype, seed=0)
    gen = torch.Generator().manual_seed(5)
    dY = torch.randn(b, T, h, p, generator=gen).to(dtype)
    r = run_operator(pkg, x, A, B, C, 128, None, dY)
    lv = [t.float().requires_grad_(True) for t in (x, A, B, C)]
    Yo, fo, co = oracle.ssd_chunked(*lv, 128)
    go = torch.autograd.grad([Yo], lv, [dY.float()])
    tol = TOL_FP32 if dtype == torch.float32 else TOL_BF16
    assert r["Y"].dtype == dtype and r["final"].dtype == dtype
    assert rel_err(r["Y"], Yo) < tol and rel_err(r["final"], fo) < tol
    for k, g in zip(("dx", "dA", "dB", "dC"), go):
        assert rel_err(r[k], g) < tol, k
    # cache contract: keys and shapes (tests/kernels/test_ssd_scan.py:99-110), values as the reference builds them
    c = T // 128
    cache = r["cache"]
    assert set(cache.keys()) == {"L", "decay_chunk", "A_cumsum"}
    assert cache["A_cumsum"].shape == (b, h, c, 128)
    assert cache["L"].shape == (b, h, c, 128, 128) and cache["decay_chunk"].shape == (b, h, c + 1, c + 1)
    assert rel_err(cache["L"], co["L"]) < tol and rel_err(cache["decay_chunk"], co["decay_chunk"]) < tol


def mamba2_gpu(pkg, inp, chunk, init=None, dfinal=None):
    leaves = {k: inp[k].detach().to(DEV).requires_grad_(True) for k in ("x", "dt", "A_head", "B", "C", "D")}
    il = init.detach().to(DEV).requires_grad_(True) if init is not None else None
    y, fs = pkg.ssd_mamba2(leaves["x"], leaves["dt"], leaves["A_head"], leaves["B"], leaves["C"], leaves["D"], chunk, il)
    outs, gouts = [y], [inp["dy"].to(DEV)]
    if dfinal is not None:
        outs.append(fs)
        gouts.append(dfinal.to(DEV))
    ins = list(leaves.values()) + ([il] if il is not None else [])
    grads = torch.autograd.grad(outs, ins, gouts)
    res = {"y": y.detach().cpu(), "final_state": fs.detach().cpu()}
    for k, g in zip(list(leaves.keys()) + (["init"] if il is not None else []), grads):
        res["d" + k] = g.detach().cpu()
    torch.cuda.synchronize()
    return res


def check_mamba2(pkg, oracle, cfg, tol, init=False, dfinal=False, seed=None):
    inp = pkg.make_inputs(cfg, seed=seed)
    g = torch.Generator().manual_seed(77)
    i0 = torch.randn(cfg.batch, cfg.nheads, cfg.headdim, cfg.d_state, generator=g) * 0.2 if init else None
    df = torch.randn(cfg.batch, cfg.nheads, cfg.headdim, cfg.d_state, generator=g) if dfinal else None
    got = mamba2_gpu(pkg, inp, cfg.chunk, i0, df)
    want = oracle.mamba2_fwd_bwd(inp, cfg.chunk, torch.float32, None if i0 is None else i0.unsqueeze(1), df)
    errs = {k: rel_err(got[k], want[k].reshape(got[k].shape)) for k in got}
    bad = {k: v for k, v in errs.items() if not v < tol}
    assert not bad, (cfg.name, errs)
    return errs


@pytest.mark.parametrize("b,T,h,at", [(1, 128, 4, (0, 0, 0)), (2, 384, 40, (1, 2, 39)), (3, 768, 36, (2, 5, 32)), (2, 1152, 66, (0, 8, 65))])
@pytest.mark.parametrize("kept", [True, False])
def test_fast_decay_in_one_block_of_the_flags(pkg, cabi, oracle, b, T, h, at, kept):
    """A log-decay of -6 a position over 40 positions of one (batch, tile, head) only, that of a block of the cumulative sums at the
    start, the end and inside the grid (heads in blocks of eight): 277 log2 units across a 32-column block, so the factorised mask of
    the backward would leave the fp32 range there.  States kept by the forward or made again."""
    bb, tile, head = at
    cfg = replace(pkg.CONFIGS[2], batch=b, seqlen=T, nheads=h, ngroups=2, chunk=128)
    inp = pkg.make_inputs(cfg, seed=17)
    inp["A_head"][head] = -60.0
    inp["dt"][:, :, head] = 1e-3
    inp["dt"][bb, tile * 128 + 50:tile * 128 + 90, head] = 0.1
    pkg.set_save_states(kept)
    try:
        got = mamba2_gpu(pkg, inp, cfg.chunk)
    finally:
        pkg.set_save_states(True)
    want = oracle.mamba2_fwd_bwd(inp, cfg.chunk, torch.float32)
    bad = {k: rel_err(got[k], want[k].reshape(got[k].shape)) for k in got if not rel_err(got[k], want[k].reshape(got[k].shape)) < TOL_BF16}
    assert not bad, bad


@pytest.mark.parametrize("h,at", [(33, (0, 0, 0)), (33, (15, 31, 32)), (36, (7, 13, 31)), (64, (3, 30, 40))])
@pytest.mark.parametrize("sums", ["kept", "made again", "given"])
def test_fast_decay_in_one_block_of_32_heads(pkg, cabi, oracle, h, at, sums):
    """The same in calls whose cumulative sums take heads in blocks of 32, where one block writes four flag words, the last one of a ragged head count fewer;
    sums from the log-decays, kept for the backward or made again by it, and given by an earlier call.  Only the batch entry with the stretch is compared."""
    bb, tile, head = at
    b, T, g = 16, 4096, 1
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=T, nheads=h, ngroups=g, chunk=64)
    gen = torch.Generator(device=DEV).manual_seed(h + tile)
    x, dy = (torch.randn(b, T, h, 64, generator=gen, device=DEV).bfloat16() for _ in range(2))
    B, C = (torch.randn(b, T, g, 128, generator=gen, device=DEV).div_(128 ** 0.5).bfloat16() for _ in range(2))
    dt, A = 0.1 * torch.rand(b, T, h, generator=gen, device=DEV), -torch.rand(h, generator=gen, device=DEV)
    A[head] = -60.0
    dt[:, :, head] = 1e-3
    dt[bb, tile * 128 + 50:tile * 128 + 90, head] = 0.1
    own = {"x": x[bb:bb + 1], "dt": dt[bb:bb + 1], "A_head": A, "B": B[bb:bb + 1], "C": C[bb:bb + 1], "D": torch.zeros(h), "dy": dy[bb:bb + 1]}
    if sums == "given":
        xs, a = (x.float() * dt.unsqueeze(-1)).bfloat16(), dt * A
        cache = pkg.fused_ssd_scan(xs[bb:bb + 1], a[bb:bb + 1], B[bb:bb + 1], C[bb:bb + 1], cfg.chunk)[2]
        full = {"A_cumsum": torch.zeros(b, h, T // cfg.chunk, cfg.chunk, device=DEV)}
        full["A_cumsum"][bb] = cache["A_cumsum"][0]
        lv = [t.requires_grad_(True) for t in (xs, B, C)]
        y = pkg.fused_ssd_scan(lv[0], a, lv[1], lv[2], cfg.chunk, None, full)[0]
        got = dict(zip(("dx", "dB", "dC"), torch.autograd.grad(y, lv, dy)), y=y)
        lo = [t[bb:bb + 1].detach().float().cpu().requires_grad_(True) for t in (xs, B, C)]
        yo = oracle.ssd_chunked(lo[0], a[bb:bb + 1].cpu(), lo[1].expand(-1, -1, h, -1), lo[2].expand(-1, -1, h, -1), cfg.chunk)[0]
        want = dict(zip(("dx", "dB", "dC"), torch.autograd.grad(yo, lo, dy[bb:bb + 1].float().cpu())), y=yo.detach())
    else:
        lv = [t.requires_grad_(True) for t in (x, dt, B, C)]
        pkg.set_save_states(sums == "kept")
        try:
            y = pkg.ssd_mamba2(lv[0], lv[1], A, lv[2], lv[3], None, cfg.chunk)[0]
            got = dict(zip(("dx", "ddt", "dB", "dC"), torch.autograd.grad(y, lv, dy)), y=y)
        finally:
            pkg.set_save_states(True)
        full = oracle.mamba2_fwd_bwd({k: v.detach().cpu() for k, v in own.items()}, cfg.chunk, torch.float32)
        want = {k: full[k] for k in got}
    bad = {k: rel_err(got[k][bb:bb + 1], want[k]) for k in got if not rel_err(got[k][bb:bb + 1], want[k]) < TOL_BF16}
    assert not bad, bad


def test_config0_fp32_full_size(pkg, cabi, oracle):
    check_mamba2(pkg, oracle, pkg.CONFIGS[0], TOL_FP32)


def test_config0_fp32_with_states(pkg, cabi, oracle):
    check_mamba2(pkg, oracle, pkg.CONFIGS[0], TOL_FP32, init=True, dfinal=True)


@pytest.mark.parametrize("path", ["simt", "tc"])
@pytest.mark.parametrize("idx,batch,seqlen", [(1, 2, 512), (2, 1, 512), (2, 2, 256)])
def test_bf16_config_shapes_reduced(pkg, cabi, oracle, idx, batch, seqlen, path):
    """Per-token shapes of the bf16 benchmark configurations at oracle-sized batch / sequence."""
    pkg.set_kernel_path(path)
    try:
        check_mamba2(pkg, oracle, pkg.shrink(pkg.CONFIGS[idx], batch, seqlen), TOL_BF16, init=(batch == 2),
                     dfinal=(batch == 2))
    finally:
        pkg.set_kernel_path("auto")


@pytest.mark.parametrize("heads,groups,batch", [(16, 2, 4), (6, 2, 4), (4, 4, 2)])
def test_tensor_core_path_with_several_items_per_cta(pkg, cabi, oracle, heads, groups, batch):
    """The backward tile kernel is persistent: with more (tile, group, batch) items than the GPU has SMs some CTAs
    process two items in a row.  8, 3 and 1 heads per group: the buffer indices and mbarrier phases carried from
    one item to the next start even, odd, and alternate every item."""
    seqlen = 128 * 20
    cfg = replace(pkg.shrink(pkg.CONFIGS[2], batch, seqlen), nheads=heads, ngroups=groups)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (seqlen // 128) * groups * batch > sms
    assert pkg.resolved_path_name(cfg) == "tc"
    check_mamba2(pkg, oracle, cfg, TOL_BF16, init=True, dfinal=True, seed=21)


@pytest.mark.parametrize("batch,seqlen,heads,groups", [(1, 128, 3, 1), (2, 256, 3, 1), (1, 128, 1, 1), (3, 384, 5, 5),
                                                       (1, 512, 6, 2), (2, 128, 9, 3), (5, 256, 7, 1), (1, 1024, 10, 2)])
@pytest.mark.parametrize("states", [False, True])
def test_tensor_core_path_edge_shapes(pkg, cabi, oracle, batch, seqlen, heads, groups, states):
    """Shapes at the edges of the tensor-core kernels' bookkeeping: one tile per sequence, one head, an odd number of
    heads per group (the double-buffered x / dy tiles and the mbarrier phases of the backward tile kernel then start an
    item on either parity, and the reverse walk runs one head per CTA), fewer work items than SMs."""
    cfg = replace(pkg.shrink(pkg.CONFIGS[2], batch, seqlen), nheads=heads, ngroups=groups)
    assert pkg.resolved_path_name(cfg) == "tc"
    check_mamba2(pkg, oracle, cfg, TOL_BF16, init=states, dfinal=states, seed=33)


@pytest.mark.parametrize("b,T,h,p,n,g,l", [(1, 1, 2, 64, 128, 1, 1), (2, 127, 3, 64, 128, 1, 127), (2, 129, 2, 64, 128, 2, 43),
                                           (2, 200, 3, 64, 128, 1, 100), (3, 320, 4, 64, 64, 2, 80), (1, 256, 2, 40, 72, 1, 64),
                                           (2, 480, 5, 56, 40, 5, 96), (1, 1300, 2, 64, 128, 1, 650)])
@pytest.mark.parametrize("states", [False, True])
def test_tensor_core_path_partial_tiles(pkg, cabi, oracle, tensor_cores, b, T, h, p, n, g, l, states):
    """Sequences that end inside a tile, chunks that end anywhere, and heads narrower than the tile's 64 x 128, on the
    tensor-core kernels when they are asked for (bar as for whole tiles: the rounding of the operands is the same)."""
    cfg = replace(pkg.CONFIGS[2], batch=b, seqlen=T, nheads=h, headdim=p, d_state=n, ngroups=g, chunk=l)
    assert pkg.resolved_path_name(cfg) == "tc"
    # (one position and no state: the decay acts on nothing, dA_head is 0 and an error relative to it is 0 / 0)
    check_mamba2(pkg, oracle, cfg, TOL_BF16, init=states or T == 1, dfinal=states, seed=77)
    inp = pkg.make_inputs(cfg, seed=78)
    a = (inp["dt"] * inp["A_head"]).to(DEV)
    args = [inp[k].to(DEV) for k in ("x", "B", "C")]
    _, _, cache = pkg.fused_ssd_scan(args[0], a, args[1], args[2], l)
    want = a.cpu().double().view(b, T // l, l, h).cumsum(2).permute(0, 3, 1, 2)
    assert rel_err(cache["A_cumsum"], want) < TOL_FP32
    y0, f0, _ = pkg.fused_ssd_scan(args[0], a, args[1], args[2], l)
    y1, f1, _ = pkg.fused_ssd_scan(args[0], a, args[1], args[2], l, None, cache)  # from the cached sums
    assert rel_err(y1, y0) < TOL_BF16 and rel_err(f1, f0) < TOL_BF16


@pytest.mark.parametrize("b,T,h,p,n,g,l", [(2, 320, 3, 64, 128, 1, 80), (2, 127, 2, 64, 128, 2, 127), (1, 256, 4, 64, 64, 2, 64),
                                           (2, 128, 2, 56, 128, 1, 64), (1, 384, 2, 64, 128, 1, 192)])
def test_partial_tiles_keep_fp32_arithmetic(pkg, cabi, oracle, b, T, h, p, n, g, l):
    """A bf16 call that does not fill whole tiles runs in fp32 unless the caller asks for the tensor cores: its fp32 outputs are
    within the fp32 bar of the oracle in fp32 on the same inputs (bf16 operands would be 2e-3 off)."""
    cfg = replace(pkg.CONFIGS[2], batch=b, seqlen=T, nheads=h, headdim=p, d_state=n, ngroups=g, chunk=l)
    assert pkg.resolved_path_name(cfg) == "simt"
    inp = pkg.make_inputs(cfg, seed=13)
    gen = torch.Generator().manual_seed(14)
    init, dfinal = torch.randn(b, h, p, n, generator=gen) * 0.2, torch.randn(b, h, p, n, generator=gen)
    got = mamba2_gpu(pkg, inp, l, init, dfinal)
    want = oracle.mamba2_fwd_bwd(inp, l, torch.float32, init.unsqueeze(1), dfinal)
    for k in ("final_state", "ddt", "dA_head", "dD", "dinit"):
        assert got[k].dtype == torch.float32 and rel_err(got[k], want[k].reshape(got[k].shape)) < TOL_FP32, k


@pytest.mark.parametrize("b,T,h,p,n,g,l", [(1, 2, 1, 64, 64, 1, 1), (2, 63, 3, 64, 72, 3, 21), (1, 65, 4, 40, 128, 2, 65), (2, 192, 8, 64, 64, 1, 96),
                                           (3, 330, 6, 56, 40, 2, 30), (8, 640, 5, 64, 64, 5, 32), (1, 448, 1, 64, 64, 1, 32), (1, 1985, 2, 40, 72, 1, 397),
                                           (2, 4090, 2, 64, 128, 1, 409),
                                           (4, 1240, 20, 64, 64, 5, 40), (1, 3008, 30, 64, 64, 5, 47), (8, 1248, 4, 64, 128, 2, 48)])
@pytest.mark.parametrize("form", ["mamba2", "operator"])
def test_partial_tiles_products_of_pieces(pkg, cabi, oracle, form, b, T, h, p, n, g, l):
    """The kernels for bf16 calls of partial tiles against the oracle in 64 bits: one position and one behind a tile, headdim and
    d_state that end inside their panels, one head per block and, in the last three, 4, 3 and 2 (on one block for the group, on two, on
    one with d_state 128), walks over the states in 1, 4 (the last
    one shorter), 11 and 16 pieces, log-decays in fp32 and bf16.  The
    three bf16 pieces of an operand carry all of its 24 bits, so what is left is the rounding of fp32 sums of at most a few
    thousand terms: 1e-5 of the largest value (two pieces would be 2^-16 off per term).  dA_head is a sum of b T signed terms
    da dt, each right to 1e-6 of the largest, and some sqrt(b T) = 72 times smaller than their absolute sum: 1e-4."""
    cfg = replace(pkg.CONFIGS[2], batch=b, seqlen=T, nheads=h, headdim=p, d_state=n, ngroups=g, chunk=l)
    base, hpg, splits = (T + 63) // 64 * b * g, h // g, 1  # blocks that share a group, as the library counts them
    while splits < hpg and (base * splits < 2 * 148 or hpg % splits):
        splits += 1
    assert hpg // splits == {1240: 4, 3008: 3, 1248: 2}.get(T, 1)
    inp = pkg.make_inputs(cfg, seed=31)
    gen = torch.Generator().manual_seed(32)
    init, dfinal = torch.randn(b, h, p, n, generator=gen) * 0.2, torch.randn(b, h, p, n, generator=gen)
    if form == "mamba2":
        got = mamba2_gpu(pkg, inp, l, init, dfinal)
        want = oracle.mamba2_fwd_bwd(inp, l, torch.float64, init.unsqueeze(1), dfinal)
        exact, rounded = ("final_state", "ddt", "dA_head", "dD", "dinit"), ("y", "dx", "dB", "dC")
    else:
        a = inp["dt"] * inp["A_head"]
        if T % 2:
            a = a.bfloat16()
        got = run_operator(pkg, inp["x"], a, inp["B"], inp["C"], l, init.unsqueeze(1), inp["dy"], dfinal.bfloat16())
        lv = [t.double().requires_grad_(True) for t in (inp["x"], a, inp["B"], inp["C"], init.unsqueeze(1))]
        Y, fs, _ = oracle.ssd_chunked(lv[0], lv[1], oracle.expand_groups(lv[2], h), oracle.expand_groups(lv[3], h), l, lv[4])
        want = dict(zip(("dx", "dA", "dB", "dC", "dinit"), torch.autograd.grad([Y, fs], lv, [inp["dy"].double(), dfinal.bfloat16().double()])), Y=Y, final=fs)
        exact, rounded = (("dA",) if a.dtype == torch.float32 else ()) + ("dinit",), ("Y", "final", "dx", "dB", "dC")
        cached = run_operator(pkg, inp["x"], a, inp["B"], inp["C"], l, init.unsqueeze(1), inp["dy"], dfinal.bfloat16(), {"A_cumsum": got["cache"]["A_cumsum"]})
        assert cached["dA"] is None and rel_err(cached["dinit"], want["dinit"].reshape(got["dinit"].shape)) < 1e-5
        for k in rounded:
            assert rel_err(cached[k], want[k].detach().reshape(got[k].shape)) < 2 ** -8, k
    for k in exact:
        assert got[k].dtype == torch.float32 and rel_err(got[k], want[k].detach().reshape(got[k].shape)) < (1e-4 if k == "dA_head" else 1e-5), k
    for k in rounded:  # one rounding to bf16
        assert rel_err(got[k], want[k].detach().reshape(got[k].shape)) < 2 ** -8, k


@pytest.mark.parametrize("case", ["state overflows", "gradient overflows", "x", "dy", "B", "C", "init", "dfinal"])
@pytest.mark.parametrize("T,n", [(192, 64), (192, 128), (40, 64), (640, 64)])
def test_partial_tiles_infinite_values(pkg, cabi, case, T, n):
    """Infinite values among the inputs, and states and their gradients that leave the range of fp32: a result that is finite, or
    infinite, with the fp32 multiply-adds of the SIMT path on the same tiles is finite, or the same infinity, here.  (An infinite value
    inside a 16-position strip: positions before it stay finite.)"""
    b, h, g, p, l = 2, 4, 2, 64, min(T, 64)
    gen = torch.Generator().manual_seed(3)
    v = {"x": torch.randn(b, T, h, p, generator=gen), "dt": 0.05 * torch.rand(b, T, h, generator=gen) + 1e-3, "A_head": -torch.exp(torch.rand(h, generator=gen)),
         "B": torch.randn(b, T, g, n, generator=gen) / n ** 0.5, "C": torch.randn(b, T, g, n, generator=gen) / n ** 0.5, "D": torch.randn(h, generator=gen),
         "init": torch.randn(b, h, p, n, generator=gen), "dy": torch.randn(b, T, h, p, generator=gen), "dfinal": torch.randn(b, h, p, n, generator=gen)}
    if case.endswith("overflows"):
        v["A_head"] *= 1e-6
        for k in ("x", "dy", "B", "C", "init", "dfinal"):  # (with both signs it would depend on the order of a sum which infinity comes first)
            v[k].abs_()
        k, m, t = ("x", "B", T // 3) if case.startswith("state") else ("dy", "C", T - 20)
        v[k][:, t], v[m][:, t] = 3e38, 30.0
    elif case in ("init", "dfinal"):
        v[case][:, 1, 5, 7], v[case][0, 2, 3] = float("inf"), float("-inf")
    else:
        v[case][:, T * 5 // 8, 1, 5], v[case][1, T // 4 + 6, 0, 6] = float("inf"), float("-inf")
    res = {}
    for path in ("auto", "simt"):
        pkg.set_kernel_path(path)
        try:
            lv = [v[k].to(DEV, torch.bfloat16 if k in "xBC" else None).requires_grad_(True) for k in ("x", "dt", "A_head", "B", "C", "D", "init")]
            y, fs = pkg.ssd_mamba2(*lv[:6], l, lv[6])
            res[path] = [y.detach(), fs.detach()] + list(torch.autograd.grad([y, fs], lv, [v["dy"].to(DEV, torch.bfloat16), v["dfinal"].to(DEV)]))
        finally:
            pkg.set_kernel_path("auto")
    infinite = 0
    for k, got, want in zip(("y", "final", "dx", "ddt", "dA_head", "dB", "dC", "dD", "dinit"), res["auto"], res["simt"]):
        inf = torch.isinf(want)
        infinite += int(inf.sum())
        assert torch.equal(got[inf], want[inf]) and torch.isfinite(got[torch.isfinite(want)]).all(), k
    assert infinite


@pytest.mark.parametrize("l", [16, 32])
def test_partial_tiles_fast_decay_in_short_chunks(pkg, cabi, oracle, l):
    """Log-decays of -0.02 to -30: what is left of a position at the end of its tile is taken from the sum of the decays behind it, not from a
    difference of sums of some hundreds (1e-5 of the state), also in the backward, where both have to agree."""
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=640, nheads=4, ngroups=1, d_state=64, chunk=l)
    inp = pkg.make_inputs(cfg, seed=3)
    inp["A_head"] = inp["A_head"] * 20
    dfinal = torch.randn(1, 4, 64, 64, generator=torch.Generator().manual_seed(5))
    got, want = mamba2_gpu(pkg, inp, l, None, dfinal), oracle.mamba2_fwd_bwd(inp, l, torch.float64, None, dfinal)
    # 64 terms of a position's own sum, each right to 2^-24 of a sum below 20 (beyond that nothing is left): 1e-6
    assert rel_err(got["final_state"], want["final_state"]) < 1e-6
    assert rel_err(got["ddt"], want["ddt"]) < 1e-5


@pytest.mark.parametrize("low", [-1e4, -1e30, -3.38e38])
@pytest.mark.parametrize("cached", [False, True])
def test_partial_tiles_resets_at_chunk_ends(pkg, cabi, oracle, low, cached):
    """Log-decays that cut the sequence off what lies before, down to the lowest values of bf16, at the last position of chunks of 16: the
    positions behind keep their own decays, whatever the kernels' tiles are.  The oracle in 64 bits gets -1000, which is as much of a cut.
    Two cuts a tile leave sums of up to 200, whose rounding of 2^-17 is what the factors between two positions are off by, twice: 2e-5."""
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=208, nheads=4, ngroups=2, d_state=64, chunk=16)
    inp = pkg.make_inputs(cfg, seed=17)
    res, a = [], inp["dt"] * inp["A_head"]
    for v in (low, -1000.0):
        a = a.clone()
        a[:, [15, 31, 143, 159]] = v
        res.append(a)
    cache = None
    if cached:
        cache = {"A_cumsum": res[0].view(1, 13, 16, 4).cumsum(2).permute(0, 3, 1, 2).contiguous().to(DEV)}
    got = run_operator(pkg, inp["x"], res[0], inp["B"], inp["C"], 16, None, inp["dy"], None, cache)
    lv = [t.double().requires_grad_(True) for t in (inp["x"], res[1], inp["B"], inp["C"])]
    Y, fs, _ = oracle.ssd_chunked(lv[0], lv[1], oracle.expand_groups(lv[2], 4), oracle.expand_groups(lv[3], 4), 16)
    want = dict(zip(("dx", "dA", "dB", "dC"), torch.autograd.grad(Y, lv, inp["dy"].double())), Y=Y, final=fs)
    for k in ("Y", "final", "dx", "dB", "dC") + (() if cached else ("dA",)):  # the others are rounded to bf16
        assert rel_err(got[k], want[k].detach().reshape(got[k].shape)) < (2e-5 if k == "dA" else 2 ** -8), k


@pytest.mark.parametrize("dtype,T,n,l", [("fp32", 192, 64, 64), ("bf16", 330, 64, 30), ("bf16", 990, 64, 30), ("bf16", 2048, 128, 128)])
def test_launch_order_eager_and_captured(pkg, cabi, dtype, T, n, l):
    """Kernels are set up while the one before them runs: the same bits call after call, on inputs and memory that the calls before
    have used, and from a captured graph, on the kernels of each path."""
    cfg = replace(pkg.CONFIGS[2], dtype=dtype, batch=2, seqlen=T, nheads=6, ngroups=2, d_state=n, chunk=l)
    inps = [{k: v.to(DEV) for k, v in pkg.make_inputs(cfg, seed=s).items()} for s in (41, 42)]
    names = ("x", "dt", "A_head", "B", "C", "D")

    def call(inp):
        lv = [inp[k].detach().requires_grad_(True) for k in names]
        y, fs = pkg.ssd_mamba2(*lv, l)
        return [y.detach(), fs.detach()] + list(torch.autograd.grad([y], lv, [inp["dy"]]))

    want = []
    for inp in inps:
        want.append([t.clone() for t in call(inp)])
        torch.cuda.synchronize()
    for i in range(20):  # back to back, in the memory of the call before
        for inp, w in zip(inps, want):
            for a, b in zip(call(inp), w):
                assert torch.equal(a, b), i
    pkg.set_check_status(False)  # (it synchronises, which a capture cannot)
    try:
        static = {k: v.clone() for k, v in inps[0].items()}
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            call(static)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = call(static)
        for inp, w in list(zip(inps, want)) * 3:
            for k in static:
                static[k].copy_(inp[k])
            graph.replay()
            for a, b in zip(outs, w):
                assert torch.equal(a, b)
    finally:
        pkg.set_check_status(True)


def test_partial_tiles_in_less_workspace(pkg, cabi):
    """With the workspace of the fp32 multiply-add kernels only (fp32 states of 96-position chunks), these run."""
    cfg = replace(pkg.CONFIGS[2], batch=2, seqlen=192, nheads=4, ngroups=2, chunk=96)
    inp = pkg.make_inputs(cfg, seed=6)
    state = 2 * 4 * 64 * 128 * 4  # of one chunk
    def up(v):
        return (v + 255) // 256 * 256
    rows, parts = up(2 * 4 * 192 * 4), up(2 * 192 * 2 * 2 * 128 * 4)
    import ctypes
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, 2, 192, 4, 64, 128, 2, 96)
    ws = {cabi.PASS_FWD: 2 * state, cabi.PASS_BWD: 5 * state + 4 * rows + 2 * 256 + 2 * parts}
    lib, res = cabi.load(), []
    for path, room in ((cabi.PATH_AUTO, None), (cabi.PATH_AUTO, ws), (cabi.PATH_SIMT, ws)):
        before = cabi.launch_count()
        res.append(_cabi_passes(pkg, cabi, cfg, inp, (), path, room) + (cabi.launch_count() - before,))
    (rc0, want, n0), (rc1, got, n1), (rc2, simt, n2) = res
    assert rc0 == rc1 == rc2 == [0, 0]
    assert n0 < n1 == n2  # 3 + 4 launches against 4 + 7
    for k in want:
        assert torch.equal(got[k], simt[k]) and rel_err(got[k], want[k]) < (1e-5 if want[k].dtype == torch.float32 else 2 ** -7), k
    assert not torch.equal(want["ddt"], simt["ddt"])
    assert [int(lib.ssd_b200_workspace_min_bytes(ctypes.byref(shape), k)) for k in sorted(ws)] == [ws[k] for k in sorted(ws)]
    rc3, _ = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO, {k: v - 1 for k, v in ws.items()})
    assert rc3 == [cabi.EWORKSPACE, cabi.EWORKSPACE]


def test_partial_tiles_where_memory_is_short(pkg, cabi):
    """With chunks of 1000 positions the pieces of the states take 24 times the room of the fp32 states of the chunks.  A call that has
    room for the latter only runs on the kernels that need no more."""
    cfg = replace(pkg.CONFIGS[2], batch=4, seqlen=4000, nheads=20, ngroups=5, chunk=1000)
    inp = {k: v.to(DEV) for k, v in pkg.make_inputs(cfg, seed=9).items()}

    def call():
        lv = [inp[k].detach().requires_grad_(True) for k in ("x", "dt", "A_head", "B", "C", "D")]
        y, fs = pkg.ssd_mamba2(*lv, cfg.chunk)
        return [y.detach(), fs.detach()] + list(torch.autograd.grad([y], lv, [inp["dy"]]))

    want = call()
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, 4, 4000, 20, 64, 128, 5, 1000)
    import ctypes
    full, least = (int(f(ctypes.byref(shape), cabi.PASS_BWD)) for f in (cabi.load().ssd_b200_workspace_bytes, cabi.load().ssd_b200_workspace_min_bytes))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = least + 200 * 2 ** 20  # the outputs and the allocator's blocks
    assert room < full
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / torch.cuda.get_device_properties(0).total_memory)
    try:
        got = call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for k, a, b in zip(("y", "final", "dx", "ddt", "dA_head", "dB", "dC", "dD"), got, want):
        assert rel_err(a, b) < (1e-4 if a.dtype == torch.float32 else 2 ** -7), k


def test_cached_call_takes_any_chunk(pkg, cabi):
    """With the sums given, nothing bounds the chunk (2048 positions of 32 heads are too many for the kernel that makes the sums,
    which is refused); same result as with chunks of 128."""
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=2048, nheads=32, ngroups=2, chunk=2048)
    inp = pkg.make_inputs(cfg, seed=4)
    a = (inp["dt"] * inp["A_head"]).to(DEV)
    x, B, C, dy = (inp[k].to(DEV) for k in ("x", "B", "C", "dy"))
    with pytest.raises(NotImplementedError, match="too large for the cumsum tile"):
        pkg.fused_ssd_scan(x, a, B, C, 2048)
    res = []
    for l in (128, 2048):
        cum = a.view(1, 2048 // l, l, 32).cumsum(2).permute(0, 3, 1, 2).contiguous()
        lv = [t.detach().requires_grad_(True) for t in (x, B, C)]
        y, fs, _ = pkg.fused_ssd_scan(lv[0], a, lv[1], lv[2], l, None, {"A_cumsum": cum})
        res.append([y.detach(), fs] + list(torch.autograd.grad([y], lv, [dy])))
    for u, v in zip(*res):
        assert rel_err(u, v) < TOL_BF16


@pytest.mark.parametrize("b,T,h,p,n,g,l", [(2, 3200, 6, 8, 16, 1, 64), (1, 128, 4, 100, 200, 2, 128), (1, 192, 2, 64, 256, 1, 96),
                                           (1, 64, 8, 65, 8, 2, 16), (2, 256, 12, 40, 65, 2, 128)])
def test_fp32_head_splits_and_wide_states(pkg, cabi, oracle, b, T, h, p, n, g, l):
    """The heads of a group on one block, on some and on one block each; states beyond 64 x 64, up to where the backward's
    panels have to share memory; several 64-row blocks per chunk with a partial last one."""
    cfg = replace(pkg.CONFIGS[0], batch=b, seqlen=T, nheads=h, headdim=p, d_state=n, ngroups=g, chunk=l)
    check_mamba2(pkg, oracle, cfg, TOL_FP32, init=True, dfinal=True, seed=99)


def _shifted(t):
    """The same values on the GPU, starting one element behind a 16-byte boundary."""
    out = torch.empty(t.numel() + 8, dtype=t.dtype, device=DEV)[1:t.numel() + 1].view(t.shape).copy_(t)
    assert out.data_ptr() % 16 and out.is_contiguous()
    return out


@pytest.mark.parametrize("T", [256, 192])
def test_unaligned_inputs(pkg, cabi, T):
    """Tensors that start between two 16-byte boundaries, through the Python operators: copied to where the kernels want them."""
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=T, nheads=2, ngroups=1, chunk=64)
    inp = pkg.make_inputs(cfg, seed=5)
    got = pkg.ssd_mamba2(_shifted(inp["x"]), inp["dt"].to(DEV), inp["A_head"].to(DEV), _shifted(inp["B"]), _shifted(inp["C"]),
                         inp["D"].to(DEV), cfg.chunk)
    want = pkg.ssd_mamba2(*[inp[k].to(DEV) for k in ("x", "dt", "A_head", "B", "C", "D")], cfg.chunk)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_segments_of_partial_tiles_take_unaligned_tensors(pkg, cabi):
    """The segmented scan hands its tensors on as they are; segments that end inside a tile run on kernels that take any address."""
    import importlib
    split = importlib.import_module("dhammic-ai_b200.distributed")
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=384, nheads=2, ngroups=1, chunk=96)
    inp = pkg.make_inputs(cfg, seed=8)
    res = []
    for place in (lambda t: t.to(DEV), _shifted):
        lv = [(place(inp[k]) if k in ("x", "B", "C") else inp[k].to(DEV)).requires_grad_(True) for k in ("x", "dt", "A_head", "B", "C", "D")]
        y, _ = split.ssd_mamba2_segmented(*lv, cfg.chunk, segments=2)
        res.append([y.detach()] + list(torch.autograd.grad([y], lv, [place(inp["dy"])])))
    for u, v in zip(*res):
        assert torch.equal(u, v)


def _cabi_passes(pkg, cabi, cfg, inp, shifted, path, ws_bytes=None):
    """Forward and backward of the Mamba-2 form straight through the C ABI, the tensors named in `shifted` off the 16-byte
    boundaries; returns (return codes, outputs)."""
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    P, st = S._ptr, S._stream(torch.device(DEV))
    b, T, h, p, n = cfg.batch, cfg.seqlen, cfg.nheads, cfg.headdim, cfg.d_state
    def place(name, t):
        return _shifted(t) if name in shifted else t.to(DEV).clone()
    t = {k: place(k, inp[k]) for k in ("x", "B", "C", "dy")}
    t.update({k: inp[k].to(DEV) for k in ("dt", "A_head", "D")})
    o = {k: place(k, torch.zeros_like(inp[v])) for k, v in (("y", "x"), ("dx", "x"), ("dB", "B"), ("dC", "C"))}
    o.update(final=torch.empty(b, h, p, n, device=DEV), cum=torch.zeros(b, h, T // cfg.chunk, cfg.chunk, device=DEV), ddt=torch.empty(b, T, h, device=DEV),
             dA_head=torch.empty(h, device=DEV), dD=torch.empty(h, device=DEV))
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16 if cfg.dtype == "bf16" else cabi.F32, cabi.F32, path, b, T, h, p, n, cfg.ngroups, cfg.chunk)
    rcs = []
    for which in (cabi.PASS_FWD, cabi.PASS_BWD):
        full = int(lib.ssd_b200_workspace_bytes(ctypes.byref(shape), which))
        ws = torch.empty(full, dtype=torch.uint8, device=DEV)
        nb = full if ws_bytes is None else ws_bytes[which]
        if which == cabi.PASS_FWD:
            a = cabi.FwdArgs(shape, P(t["x"]), None, P(t["dt"]), P(t["A_head"]), P(t["D"]), P(t["B"]), P(t["C"]), None, P(o["y"]), P(o["final"]),
                             P(o["cum"]), 0, 0, P(ws), nb)
            rcs.append(lib.ssd_b200_fwd(ctypes.byref(a), st))
        else:
            a = cabi.BwdArgs(shape, P(t["x"]), None, P(t["dt"]), P(t["A_head"]), P(t["D"]), P(t["B"]), P(t["C"]), None, P(o["cum"]), P(t["dy"]), None,
                             P(o["dx"]), P(o["dB"]), P(o["dC"]), None, P(o["ddt"]), P(o["dA_head"]), P(o["dD"]), None, 0, 0, P(ws), nb)
            rcs.append(lib.ssd_b200_bwd(ctypes.byref(a), st))
        torch.cuda.synchronize()
    return rcs, o


@pytest.mark.parametrize("shifted", [("x",), ("B", "C"), ("y",), ("dy", "dx"), ("dB",), ("x", "B", "C", "y", "dy", "dx", "dB", "dC")])
@pytest.mark.parametrize("dtype,n,g", [("bf16", 128, 2), ("bf16", 64, 4), ("bf16", 128, 4), ("fp32", 128, 2)])
def test_unaligned_tensors_through_the_c_abi(pkg, cabi, dtype, n, g, shifted):
    """The SIMT kernels and those for partial tiles (d_state 64 and 128, dB and dC from one block and from several) take any address: the same
    bits as with aligned tensors.  The tcgen05 kernels refuse on the host."""
    cfg = replace(pkg.CONFIGS[2], dtype=dtype, batch=2, seqlen=192, nheads=4, ngroups=g, d_state=n, chunk=64)
    inp = pkg.make_inputs(cfg, seed=6)
    rc0, want = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO)
    rc1, got = _cabi_passes(pkg, cabi, cfg, inp, shifted, cabi.PATH_AUTO)
    assert rc0 == rc1 == [0, 0]
    for k in want:
        assert torch.equal(want[k], got[k]), k
    if dtype == "bf16" and n == 128:
        whole = replace(cfg, seqlen=256)
        rcs, _ = _cabi_passes(pkg, cabi, whole, pkg.make_inputs(whole, seed=6), shifted, cabi.PATH_AUTO)
        refused = [bool({"x", "B", "C", "y"} & set(shifted)), bool({"x", "B", "C", "dy", "dx", "dB", "dC"} & set(shifted))]
        assert [rc == cabi.EINVAL for rc in rcs] == refused


@pytest.mark.parametrize("b,T,h,g", [(1, 4096, 64, 2), (1, 4480, 64, 8), (2, 3968, 36, 3), (1, 4096, 64, 32)])
def test_reverse_walk_in_pieces_of_two_heads(pkg, cabi, b, T, h, g):
    """Sequences whose reverse walk is cut into pieces with two heads of a group per CTA (whole last pieces and short ones, two heads per group): the same
    as in one piece, which is what a call with room for no more takes.  States and gradients are bf16 sums of the same terms in another order.  The
    summaries launched say what was cut: the forward's walk, the same walk in the backward, and the reverse one."""
    import ctypes
    cfg = replace(pkg.CONFIGS[2], batch=b, seqlen=T, nheads=h, ngroups=g, chunk=128)
    inp = pkg.make_inputs(cfg, seed=8)
    def up(v):
        return (v + 255) // 256 * 256
    nt, bh = T // 128, b * h
    bht, state = up(bh * T * 4), up(bh * 64 * 128 * 4)
    fwd = 256 + 3 * bht
    bwd = fwd + 2 * up(bh * nt * 64 * 128 * 2) + 2 * state + 3 * bht + up(bh * nt * 32) + 2 * up(bh * nt * 4)
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, b, T, h, 64, 128, g, 128)
    assert cabi.load().ssd_b200_workspace_bytes(ctypes.byref(shape), cabi.PASS_BWD) > bwd
    def passes(*room):
        cabi.profile_enable(True)
        try:
            rcs, out = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO, *room)
            return rcs, out, cabi.profile_read().get("tc_summary", (0.0, 0))[1]
        finally:
            cabi.profile_enable(False)
    rc0, want, whole = passes({cabi.PASS_FWD: fwd, cabi.PASS_BWD: bwd})
    rc1, got, cut = passes()
    assert rc0 == rc1 == [0, 0] and (whole, cut) == (0, 3)
    for k in want:
        assert rel_err(got[k], want[k]) < TOL_BF16, k


@pytest.mark.parametrize("T,h,g", [(6144, 96, 2), (12288, 128, 8), (24576, 76, 1)])
def test_gradients_of_many_heads_do_not_depend_on_the_batch(pkg, cabi, T, h, g):
    """One batch entry of 75 to 148 (batch, head) pairs alone, and the same entry in a batch of two: outputs and gradients have the same bits, so a call
    may be cut into micro-batches (with fewer pairs the walks are cut into pieces, and with them the sums)."""
    cfg = replace(pkg.CONFIGS[2], batch=2, seqlen=T, nheads=h, ngroups=g, chunk=128)
    gen = torch.Generator(device=DEV).manual_seed(T)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    x, B, C, dy = (randn(2, T, *s).bfloat16() for s in ((h, 64), (g, 128), (g, 128), (h, 64)))
    dt, A, D = 0.05 * torch.rand(2, T, h, generator=gen, device=DEV), -torch.rand(h, generator=gen, device=DEV), randn(h)
    def run(part):
        lv = [t.requires_grad_(True) for t in (x[part].clone(), dt[part].clone(), A.clone(), B[part].clone() / 128 ** 0.5, C[part].clone(), D.clone())]
        y, fs = pkg.ssd_mamba2(*lv, cfg.chunk)
        return [y, fs, *(v for i, v in enumerate(torch.autograd.grad(y, lv, dy[part])) if i not in (2, 5))]
    whole = run(slice(None))
    for i in range(2):
        for name, u, v in zip(("y", "final", "dx", "ddt", "dB", "dC"), run(slice(i, i + 1)), whole):
            assert torch.equal(u, v[i:i + 1]), name


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 6, 9, 12])
@pytest.mark.parametrize("h,g,few,many", [(1, 1, 1, 80), (3, 1, 2, 27), (6, 2, 4, 14), (3, 1, 56, 28)])
def test_walks_that_find_their_own_way(pkg, cabi, tiles, h, g, few, many):
    """Forward walks that leave most SMs idle (all of a call's, or those behind the last full round of 148) are cut, and every CTA makes the states before its tiles
    for itself: outputs, states and the norm's statistic have the bits of whole walks, which calls of 75 to 148 pairs take.  Lengths from
    one tile to the longest whose walks are not summarised instead; with and without per-position arrays and kept states."""
    T, n = 128 * tiles, max(few, many)
    gen = torch.Generator(device=DEV).manual_seed(tiles)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    x, z, B, C = (randn(n, T, *s).bfloat16() for s in ((h, 64), (h * 64,), (g, 128), (g, 128)))
    dt, A, D, w = 0.05 * torch.rand(n, T, h, generator=gen, device=DEV), -torch.rand(h, generator=gen, device=DEV), randn(h), randn(h * 64)
    init = randn(n, h, 64, 128)
    def run(b):
        xb, zb, Bb, Cb, dtb, ib = (t[:b].contiguous() for t in (x, z, B / 128 ** 0.5, C, dt, init))
        out = [*pkg.ssd_mamba2(xb, dtb, A, Bb, Cb, D, 128, ib), *pkg.ssd_mamba2_gated(xb, dtb, A, Bb, Cb, None, zb, w, 1e-6, 128),
               *pkg.fused_ssd_scan(xb, (dtb * A), Bb, Cb, 128)[:2]]
        leaf = xb.clone().requires_grad_(True)  # with the states kept for the backward
        y, fs = pkg.ssd_mamba2(leaf, dtb, A, Bb, Cb, D, 128, ib)
        return out + [y.detach(), fs.detach(), torch.autograd.grad(y, leaf, xb)[0]]
    m = min(few, many)
    for i, (u, v) in enumerate(zip(run(few), run(many))):
        # (the gradient of few pairs takes another reverse walk, and the states are what the walks left)
        assert torch.equal(u[:m], v[:m]) if i < 8 else rel_err(u[:m].float(), v[:m].float()) < TOL_BF16, i


@pytest.mark.parametrize("tiles", [2, 5, 12, 40])
@pytest.mark.parametrize("h,g,batch", [(3, 1, 56), (24, 1, 8), (4, 2, 40)])
def test_walks_behind_a_full_round(pkg, cabi, tiles, h, g, batch):
    """Of 160 to 192 forward walks those behind the first 148 are cut (in up to four pieces); the last entries of the batch, on both sides of that line, have the bits
    that they have in a call of their own, of 75 and more walks, which are whole."""
    T, n = 128 * tiles, -(-75 // h)
    assert batch * h > 148 and (batch - n) * h < 148
    gen = torch.Generator(device=DEV).manual_seed(tiles)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    x, z, B, C = (randn(batch, T, *s).bfloat16() for s in ((h, 64), (h * 64,), (g, 128), (g, 128)))
    dt, A, D, w = 0.05 * torch.rand(batch, T, h, generator=gen, device=DEV), -torch.rand(h, generator=gen, device=DEV), randn(h), randn(h * 64)
    init = randn(batch, h, 64, 128)
    def run(first):
        xb, zb, Bb, Cb, dtb, ib = (t[first:].contiguous() for t in (x, z, B / 128 ** 0.5, C, dt, init))
        leaf = xb.clone().requires_grad_(True)  # with the states kept for the backward
        y, fs = pkg.ssd_mamba2(leaf, dtb, A, Bb, Cb, D, 128, ib)
        return [*pkg.ssd_mamba2(xb, dtb, A, Bb, Cb, D, 128, ib), *pkg.ssd_mamba2_gated(xb, dtb, A, Bb, Cb, None, zb, w, 1e-6, 128),
                *pkg.fused_ssd_scan(xb, dtb * A, Bb, Cb, 128)[:2], y.detach(), fs.detach(), torch.autograd.grad(y, leaf, xb)[0]]
    for i, (u, v) in enumerate(zip(run(0), run(batch - n))):
        assert torch.equal(u[batch - n:], v), i


_FIRST_BACKWARD = """
import sys
sys.path.insert(0, {root!r})
import importlib, torch
pkg = importlib.import_module("dhammic-ai_b200")
cfg = pkg.shrink(pkg.CONFIGS[2], 1, 256)
inp = pkg.make_inputs(cfg)
names = ("x", "dt", "A_head", "B", "C", "D")
lv = [inp[k].cuda().requires_grad_(True) for k in names]
dy = inp["dy"].cuda()
side = torch.cuda.Stream()
torch.cuda.synchronize()
with torch.cuda.stream(side):  # (a backward runs on its forward's stream)
    y, _ = pkg.ssd_mamba2(*lv, cfg.chunk)
    room = [torch.empty(64 << 20, dtype=torch.uint8, device="cuda")] + [torch.empty(512, device="cuda") for _ in range(600)]
    del room
torch.cuda.synchronize()
if {capture}:
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        first = torch.autograd.grad([y], lv, [dy], retain_graph=True)
    graph.replay()
else:
    with torch.cuda.stream(side):
        first = torch.autograd.grad([y], lv, [dy], retain_graph=True)
torch.cuda.synchronize()
with torch.cuda.stream(side):
    again = torch.autograd.grad([y], lv, [dy])
torch.cuda.synchronize()
assert all(torch.equal(u, v) for u, v in zip(first, again))
print("same")
"""


@pytest.mark.parametrize("capture", [False, True])
def test_first_backward_of_a_process(pkg, cabi, capture):
    """The first backward, on an autograd thread that has not called the runtime yet and needs a context for its tensor maps: with room in the allocator, so that no
    allocation binds one before, and inside a capture, where what binds it must be allowed.  In a process of its own, since only the first is of interest."""
    import subprocess
    import sys
    from pathlib import Path
    code = _FIRST_BACKWARD.format(root=str(Path(__file__).resolve().parents[1]), capture=capture)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]


def test_walk_in_one_piece_where_the_workspace_has_no_room(pkg, cabi):
    """With less workspace than several pieces need, but enough for one, the walks run in one; with a byte less they are refused."""
    cfg = replace(pkg.CONFIGS[2], batch=1, seqlen=4096, nheads=6, ngroups=2, chunk=128)
    inp = pkg.make_inputs(cfg, seed=7)
    lib = cabi.load()
    import ctypes
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, 1, 4096, 6, 64, 128, 2, 128)
    def up(v):
        return (v + 255) // 256 * 256
    nt, bht, state = 32, up(6 * 4096 * 4), up(6 * 64 * 128 * 4)
    fwd = 256 + 3 * bht
    bwd = fwd + 2 * up(6 * nt * 64 * 128 * 2) + 2 * state + 3 * bht + up(6 * nt * 32) + 2 * up(6 * nt * 4)
    assert lib.ssd_b200_workspace_bytes(ctypes.byref(shape), cabi.PASS_FWD) > fwd
    assert lib.ssd_b200_workspace_bytes(ctypes.byref(shape), cabi.PASS_BWD) > bwd
    rc0, want = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO)
    rc1, got = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO, {cabi.PASS_FWD: fwd, cabi.PASS_BWD: bwd})
    assert rc0 == rc1 == [0, 0]
    for k in want:
        assert rel_err(got[k], want[k]) < TOL_BF16, k
    rc2, _ = _cabi_passes(pkg, cabi, cfg, inp, (), cabi.PATH_AUTO, {cabi.PASS_FWD: fwd - 1, cabi.PASS_BWD: bwd - 1})
    assert rc2 == [cabi.EWORKSPACE, cabi.EWORKSPACE]


@pytest.mark.parametrize("dtype,b,T,h,n,g", [("bf16", 1, 512, 24, 128, 1), ("bf16", 1, 1024, 64, 128, 8), ("bf16", 8, 512, 24, 128, 1), ("bf16", 1, 8192, 8, 128, 2),
                                             ("bf16", 1, 4032, 4, 64, 1), ("bf16", 1, 4032, 4, 128, 1), ("fp32", 2, 256, 8, 64, 1)])
def test_state_updated_in_place(pkg, cabi, dtype, b, T, h, n, g):
    """init and final_state in one buffer: the results of two.  Walks that are cut where the two are apart (by themselves, summarised, those of partial tiles, behind a
    full round) and whole ones.  On the tcgen05 kernels the bits are those of a call with room for one piece."""
    cfg = replace(pkg.CONFIGS[2], dtype=dtype, batch=b, seqlen=T, nheads=h, ngroups=g, d_state=n, chunk=64)
    inp = {k: v.to(DEV) for k, v in pkg.make_inputs(cfg, seed=6).items()}
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    P, st = S._ptr, S._stream(torch.device(DEV))
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16 if dtype == "bf16" else cabi.F32, cabi.F32, cabi.PATH_AUTO, b, T, h, 64, n, g, 64)
    tc = lib.ssd_b200_resolve_path(ctypes.byref(shape)) == cabi.PATH_TC
    room = {f: int(getattr(lib, f"ssd_b200_workspace_{f}")(ctypes.byref(shape), cabi.PASS_FWD)) for f in ("bytes", "min_bytes")}
    ws, init = torch.empty(room["bytes"], dtype=torch.uint8, device=DEV), torch.randn(b, h, 64, n, device=DEV)
    def run(in_place, nb):
        state, y, cum = init.clone(), torch.empty_like(inp["x"]), torch.empty(b, h, T // 64, 64, device=DEV)
        final = state if in_place else torch.empty_like(init)
        a = cabi.FwdArgs(shape, P(inp["x"]), None, P(inp["dt"]), P(inp["A_head"]), P(inp["D"]), P(inp["B"]), P(inp["C"]), P(state), P(y), P(final), P(cum), 0, 0, P(ws), nb)
        cabi.check(lib.ssd_b200_fwd(ctypes.byref(a), st))
        torch.cuda.synchronize()
        return y, final
    want = run(False, room["min_bytes" if tc else "bytes"])
    for _ in range(8):
        for u, v in zip(run(True, room["bytes"]), want):
            assert torch.equal(u, v) if tc else rel_err(u.float(), v.float()) < (1e-5 if u.dtype == torch.float32 else 2 ** -7)


@pytest.mark.parametrize("h,p,n,g,l,T", [(3, 24, 12, 1, 32, 96), (4, 80, 40, 2, 48, 96), (6, 16, 72, 3, 100, 200),
                                         (2, 128, 130, 1, 64, 64), (2, 8, 8, 2, 16, 16)])
def test_ragged_shapes_fp32(pkg, cabi, oracle, h, p, n, g, l, T):
    """Sizes that are not multiples of the 64-wide tiles, odd head/group counts, a single chunk."""
    cfg = replace(pkg.CONFIGS[0], batch=2, seqlen=T, nheads=h, headdim=p, d_state=n, ngroups=g, chunk=l)
    check_mamba2(pkg, oracle, cfg, TOL_FP32, init=True, dfinal=True, seed=4242)


def test_sequence_split_through_states(pkg, cabi, oracle):
    """Two halves chained through final_state -> initial_states reproduce the full run (fwd and grads)."""
    cfg = pkg.shrink(pkg.CONFIGS[0], batch=1, seqlen=256)
    inp = pkg.make_inputs(cfg)
    full = mamba2_gpu(pkg, inp, cfg.chunk)
    lo = {k: (v[:, :128] if v.dim() >= 3 else v) for k, v in inp.items()}
    hi = {k: (v[:, 128:] if v.dim() >= 3 else v) for k, v in inp.items()}
    first = mamba2_gpu(pkg, lo, cfg.chunk)
    second = mamba2_gpu(pkg, hi, cfg.chunk, init=first["final_state"])
    assert rel_err(torch.cat([first["y"], second["y"]], 1), full["y"]) < TOL_FP32
    assert rel_err(second["final_state"], full["final_state"]) < TOL_FP32
    # backward: the second half's d_init is the first half's dfinal
    first_b = mamba2_gpu(pkg, lo, cfg.chunk, dfinal=second["dinit"])
    assert rel_err(torch.cat([first_b["dx"], second["dx"]], 1), full["dx"]) < TOL_FP32
    assert rel_err(torch.cat([first_b["ddt"], second["ddt"]], 1), full["ddt"]) < TOL_FP32
    assert rel_err(first_b["dA_head"] + second["dA_head"], full["dA_head"]) < TOL_FP32


def test_error_behaviour_on_gpu(pkg, cabi):
    x = torch.zeros(1, 100, 2, 8, device=DEV)
    A = torch.zeros(1, 100, 2, device=DEV)
    B = torch.zeros(1, 100, 2, 4, device=DEV)
    with pytest.raises(AssertionError, match="not divisible"):
        pkg.fused_ssd_scan(x, A, B, B, 64)
    with pytest.raises(RuntimeError, match="same dtype"):
        pkg.fused_ssd_scan(x[:, :64], A[:, :64], B[:, :64].bfloat16(), B[:, :64], 64)


def _scan_args(b=2, T=128, h=2, p=64, n=128, g=1, dtype=torch.bfloat16):
    gen = torch.Generator(device=DEV).manual_seed(b + T + h)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    return {"x": randn(b, T, h, p).to(dtype), "dt": 0.1 * torch.rand(b, T, h, generator=gen, device=DEV), "A_head": -torch.ones(h, device=DEV),
            "B": (0.1 * randn(b, T, g, n)).to(dtype), "C": (0.1 * randn(b, T, g, n)).to(dtype), "D": randn(h)}


def _call(pkg, op, a):
    if op == "mamba2":
        return pkg.ssd_mamba2(*[a[k] for k in ("x", "dt", "A_head", "B", "C", "D")], 64, a.get("init"))
    if op == "operator":
        cache = {"A_cumsum": a["cum"]} if "cum" in a else None
        return pkg.fused_ssd_scan(a["x"], a["dt"], a["B"], a["C"], 64, a.get("init"), cache)[:2]
    if op == "gated":
        return pkg.ssd_mamba2_gated(*[a[k] for k in ("x", "dt", "A_head", "B", "C", "D", "z", "weight")], 1e-6, 64, a.get("init"))
    return (pkg.ssd_mamba3(*[a[k] for k in ("x", "dt", "A_head", "B", "C", "D", "angles", "lam")], 64),)


def _op_args(op, **kw):
    a = _scan_args(**kw)
    b, T, h, p = a["x"].shape
    n = a["B"].shape[3]
    if op == "gated":
        a.update(z=torch.ones(b, T, h * p, dtype=a["x"].dtype, device=DEV), weight=torch.ones(h * p, device=DEV))
    if op == "mamba3":
        a.update(angles=torch.ones(b, T, h, n // 2, dtype=a["x"].dtype, device=DEV), lam=torch.full((b, T, h), 0.5, device=DEV))
    return a


@pytest.mark.parametrize("op,arg,bad", [
    ("mamba2", "dt", (2, 64, 2)), ("mamba2", "A_head", (1,)), ("mamba2", "D", (1,)), ("mamba2", "init", (1, 2, 64, 128)), ("mamba2", "dt", "cpu"),
    ("operator", "dt", (2, 128, 1)), ("operator", "init", (2, 1, 2, 64, 64)), ("operator", "cum", (2, 2, 1, 64)), ("operator", "cum", "cpu"),
    ("gated", "weight", (64,)), ("gated", "weight", "cpu"), ("gated", "z", (2, 128, 64)), ("gated", "A_head", (1,)),
    ("mamba3", "angles", (2, 128, 2, 32)), ("mamba3", "lam", (2, 64, 2)), ("mamba3", "D", (1,)), ("mamba3", "dt", (2, 128, 1)), ("mamba3", "angles", "cpu"),
    ("mamba3", "C", (2, 128, 1, 64)), ("mamba3", "B", "fp32")])
def test_arguments_that_are_too_small_are_refused(pkg, cabi, op, arg, bad):
    """Kernels read these by x's sizes: what is shorter, of another type or on another device ends in an exception before any launch."""
    a = _op_args(op)
    good = a.get(arg, torch.zeros(2, 2, 2, 64, device=DEV))
    a[arg] = good.cpu() if bad == "cpu" else good.float() if bad == "fp32" else torch.zeros(*bad, dtype=good.dtype, device=DEV)
    before = cabi.launch_count()
    with pytest.raises((ValueError, AssertionError, RuntimeError)):
        _call(pkg, op, a)
    assert cabi.launch_count() == before


def test_cache_can_be_pickled_and_copied(pkg, cabi):
    """The operator's cache goes through pickle and copy before anything was read from it, and works as the one it came from."""
    import copy
    import pickle
    a = _op_args("operator", p=16, n=8, dtype=torch.float32)
    decay = -a["dt"]
    y0, _, cache = pkg.fused_ssd_scan(a["x"], decay, a["B"], a["C"], 64)
    for other in (pickle.loads(pickle.dumps(cache)), copy.copy(cache), copy.deepcopy(cache)):
        y1, _, _ = pkg.fused_ssd_scan(a["x"], decay, a["B"], a["C"], 64, None, other)
        assert torch.equal(y0, y1)
        for k in ("A_cumsum", "L", "decay_chunk"):
            assert torch.equal(other[k], cache[k])


def test_cached_sums_leave_without_their_graph(pkg, cabi):
    """Sums that the caller made with a graph are values here: the cache that comes back does not carry the graph on."""
    a = _op_args("operator")
    decay = (-a["dt"]).requires_grad_(True)
    cum = decay.view(2, 2, 64, 2).cumsum(2).permute(0, 3, 1, 2).contiguous()
    _, _, cache = pkg.fused_ssd_scan(a["x"], decay, a["B"], a["C"], 64, None, {"A_cumsum": cum})
    assert cum.requires_grad and not cache["A_cumsum"].requires_grad and torch.equal(cache["A_cumsum"], cum)


def test_status_check_holds_for_the_backward_of_earlier_forwards(pkg, cabi):
    """set_check_status is read when a pass runs: a backward of a graph recorded before synchronises (as its forward would)."""
    try:
        pkg.set_check_status(False)
        lv, out, g = _graph(pkg, "mamba2")
        pkg.set_check_status(True)
        torch.cuda.synchronize()
        spin = torch.cuda.Event()
        torch.cuda._sleep(200_000_000)  # about 0.1 s of waiting in front of the backward
        spin.record()
        torch.autograd.grad([out], lv, [g])
        assert spin.query()
    finally:
        pkg.set_check_status(True)


def _graph(pkg, op):
    """The leaves, the output and an output gradient of one call of an operator with a recorded graph."""
    if op in ("mamba2", "operator", "gated", "mamba3"):
        a = _op_args(op)
        lv = [t.requires_grad_(True) for t in a.values()] if op != "operator" else [a[k].requires_grad_(True) for k in ("x", "dt", "B", "C")]
        out = _call(pkg, op, a)[0]
    else:
        gen = torch.Generator(device=DEV).manual_seed(8)
        x = torch.randn(2, 64, 4, 16, generator=gen, device=DEV)
        lv = {"rope": [x, x[..., :8].clone()], "norm": [x, torch.ones(16, device=DEV), x.clone()],
              "trapezoid": [x[..., 0].clone(), x[..., 1].clone(), x[0, 0, :, 2].clone(), x[0, 0, :, 3].clone()]}[op]
        lv = [t.requires_grad_(True) for t in lv]
        out = {"rope": lambda: pkg.fused_rope(*lv), "norm": lambda: pkg.fused_gate_norm(lv[0], lv[2], lv[1]),
               "trapezoid": lambda: pkg.fused_trapezoidal(*lv)[2]}[op]()
    return lv, out, torch.ones_like(out)


ALL_OPS = ["mamba2", "operator", "gated", "mamba3", "rope", "norm", "trapezoid"]


@pytest.mark.parametrize("op", ALL_OPS)
def test_backward_twice_through_a_freed_graph_raises(pkg, cabi, op):
    lv, out, g = _graph(pkg, op)
    first = torch.autograd.grad([out], lv, [g], retain_graph=True, allow_unused=True)
    second = torch.autograd.grad([out], lv, [g], allow_unused=True)
    for a, b in zip(first, second):
        assert (a is None and b is None) or torch.equal(a, b)
    with pytest.raises(RuntimeError, match="backward through the graph a second time"):
        torch.autograd.grad([out], lv, [g], allow_unused=True)


@pytest.mark.parametrize("op", ALL_OPS)
def test_two_threads_on_one_graph(pkg, cabi, op):
    """Threads that run backward through one graph at the same time, one of them freeing it: each ends with the gradients or with
    torch's error about a freed graph, never with anything else."""
    import threading
    for _ in range(5):
        lv, out, g = _graph(pkg, op)
        want = torch.autograd.grad([out], lv, [g], retain_graph=True, allow_unused=True)
        got, start = {}, threading.Barrier(2)
        def work(i):
            start.wait()
            try:
                got[i] = torch.autograd.grad([out], lv, [g], retain_graph=i == 0, allow_unused=True)
                torch.cuda.synchronize()
            except RuntimeError as e:
                got[i] = e
        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i, r in got.items():
            if isinstance(r, Exception):
                assert i == 0 and "second time" in str(r)
            else:
                for a, b in zip(r, want):
                    assert (a is None and b is None) or torch.equal(a, b)


@pytest.mark.parametrize("op", ALL_OPS)
@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.filterwarnings("ignore:.*torch.jit.*:DeprecationWarning")
def test_trace_replays_the_operator(pkg, cabi, op):
    """A traced call gives on other inputs what the operator gives on them, with its gradients."""
    if op in ("mamba2", "operator", "gated", "mamba3"):
        a = _op_args(op)
        if op == "operator":
            a = {k: a[k] for k in ("x", "dt", "B", "C")}
        names = list(a)
        def fn(*t):
            return _call(pkg, op, dict(zip(names, t)))[0]
        args = list(a.values())
    else:
        lv, _, _ = _graph(pkg, op)
        args = [t.detach() for t in lv]
        fn = {"rope": pkg.fused_rope, "norm": lambda x, w, z: pkg.fused_gate_norm(x, z, w), "trapezoid": lambda *t: pkg.fused_trapezoidal(*t)[2]}[op]
    traced = torch.jit.trace(fn, tuple(args))
    gen = torch.Generator(device=DEV).manual_seed(3)
    other = [(t * (0.5 + torch.rand(t.shape, generator=gen, device=DEV))).to(t.dtype) for t in args]
    res = []
    for f in (fn, traced):
        lv = [t.clone().requires_grad_(True) for t in other]
        y = f(*lv)
        res.append([y.detach()] + list(torch.autograd.grad([y], lv, [torch.ones_like(y)], allow_unused=True)))
    for u, v in zip(*res):
        assert (u is None and v is None) or torch.equal(u, v)


def test_gated_norm_weight_per_head(pkg, cabi):
    """A weight of shape (heads, headdim) is the flat one, forward and backward (its gradient has its shape)."""
    a = _op_args("gated", h=3)
    gen = torch.Generator(device=DEV).manual_seed(1)
    w = torch.rand(3, 64, generator=gen, device=DEV)
    res = []
    for weight in (w.flatten(), w):
        a["weight"] = weight.clone().requires_grad_(True)
        a["x"] = a["x"].detach().requires_grad_(True)
        out = _call(pkg, "gated", a)[0]
        res.append([out.detach()] + list(torch.autograd.grad(out.float().square().sum(), [a["weight"], a["x"]])))
    assert res[1][1].shape == (3, 64)
    for u, v in zip(*res):
        assert torch.equal(u.flatten(), v.flatten())


def test_noncontiguous_inputs_and_determinism(pkg, cabi):
    """The caller passes products and padded views (src/mamba_base_engine.py:170-181); results are
    bitwise reproducible run to run."""
    x, A, B, C = pkg.make_reference_test_inputs(2, 256, 4, 16, 8, torch.float32, seed=3)
    xv = torch.cat([x, x], -1).to(DEV)[..., :16]
    Bv = B.to(DEV).transpose(1, 2).contiguous().transpose(1, 2)
    assert not xv.is_contiguous() and not Bv.is_contiguous()
    outs = []
    for _ in range(2):
        xl = xv.detach().requires_grad_(True)
        Al = A.to(DEV).requires_grad_(True)
        Y, fs, _ = pkg.fused_ssd_scan(xl, Al, Bv, C.to(DEV), 128)
        gx, gA = torch.autograd.grad([Y], [xl, Al], [torch.ones_like(Y)])
        outs.append((Y, fs, gx, gA))
    Yc, fc, _ = pkg.fused_ssd_scan(x.to(DEV), A.to(DEV), B.to(DEV), C.to(DEV), 128)
    assert torch.equal(outs[0][0], Yc) and torch.equal(outs[0][1], fc)
    for a, b in zip(outs[0], outs[1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("chunk", [64, 128, 256])
@pytest.mark.parametrize("a_dtype", [torch.bfloat16, torch.float32])
def test_tensor_core_path_operator_form(pkg, cabi, oracle, chunk, a_dtype):
    """fused_ssd_scan on the tcgen05 kernels (one head per group, as the reference caller uses it):
    forward, all gradients, initial/final state, and the cached second call."""
    b, T, h, p, n = 2, 512, 3, 64, 128
    x, A, B, C = pkg.make_reference_test_inputs(b, T, h, p, n, torch.bfloat16, seed=11)
    A = (A.float() * 3.0).to(a_dtype)
    gen = torch.Generator().manual_seed(12)
    dY = torch.randn(b, T, h, p, generator=gen).bfloat16()
    init = (torch.randn(b, 1, h, p, n, generator=gen) * 0.3).bfloat16()
    dfinal = torch.randn(b, h, p, n, generator=gen).bfloat16()
    pkg.set_kernel_path("tc")
    try:
        r = run_operator(pkg, x, A, B, C, chunk, init, dY, dfinal)
        x2 = torch.nn.functional.pad(x[:, :-1], (0, 0, 0, 0, 1, 0))
        B2 = torch.nn.functional.pad(B[:, :-1], (0, 0, 0, 0, 1, 0))
        r2 = run_operator(pkg, x2, A, B2, C, chunk, None, dY, None, cache=r["cache"])
    finally:
        pkg.set_kernel_path("auto")
    lv = [t.float().requires_grad_(True) for t in (x, A, B, C)]
    il = init.float().requires_grad_(True)
    Yo, fo, co = oracle.ssd_chunked(*lv, chunk, il)
    go = torch.autograd.grad([Yo, fo], lv + [il], [dY.float(), dfinal.float()])
    errs = {"Y": rel_err(r["Y"], Yo), "final": rel_err(r["final"], fo)}
    for k, g in zip(("dx", "dA", "dB", "dC", "dinit"), go):
        errs[k] = rel_err(r[k], g)
    l2 = [t.float().requires_grad_(True) for t in (x2, A, B2, C)]
    Y2, _, _ = oracle.fused_ssd_scan_oracle(*l2, chunk, None, co)
    g2 = torch.autograd.grad([Y2], [l2[0], l2[2], l2[3]], [dY.float()])
    errs["Y_cached"] = rel_err(r2["Y"], Y2)
    for k, g in zip(("dx", "dB", "dC"), g2):
        errs[k + "_cached"] = rel_err(r2[k], g)
    assert r2["dA"] is None
    bad = {k: v for k, v in errs.items() if not v < TOL_BF16}
    assert not bad, errs


def test_tensor_core_path_is_deterministic_and_selected(pkg, cabi):
    cfg = pkg.shrink(pkg.CONFIGS[2], 2, 512)
    assert pkg.resolved_path_name(cfg) == "tc"
    assert pkg.resolved_path_name(pkg.CONFIGS[0]) == "simt"
    inp = pkg.make_inputs(cfg)
    a = mamba2_gpu(pkg, inp, cfg.chunk)
    b = mamba2_gpu(pkg, inp, cfg.chunk)
    for k in a:
        assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("chunk", [128, 64, 32, 256, 512])
def test_saved_states_equal_recomputed_states(pkg, cabi, chunk):
    """The backward gives the same gradients whether the forward kept its per-tile states or the
    backward recomputes them (the reference's input-only checkpointing)."""
    cfg = replace(pkg.shrink(pkg.CONFIGS[2], 2, 512), chunk=chunk)
    inp = pkg.make_inputs(cfg)
    g = torch.Generator().manual_seed(9)
    init = torch.randn(cfg.batch, cfg.nheads, cfg.headdim, cfg.d_state, generator=g) * 0.2
    kept = mamba2_gpu(pkg, inp, cfg.chunk, init)
    pkg.set_save_states(False)
    try:
        redone = mamba2_gpu(pkg, inp, cfg.chunk, init)
    finally:
        pkg.set_save_states(True)
    for k in kept:
        assert torch.equal(kept[k], redone[k]), k


@pytest.mark.parametrize("b,T,h,g,p,n,chunk", [(1, 4096, 6, 2, 64, 128, 128), (1, 3008, 30, 5, 64, 64, 64), (2, 6016, 4, 4, 48, 128, 64),
                                               (1, 16384, 9, 1, 64, 128, 256), (1, 6016, 56, 8, 64, 128, 128)])
def test_walks_in_pieces(pkg, cabi, oracle, tensor_cores, b, T, h, g, p, n, chunk):
    """Few (batch, head) pairs and a long sequence: the walks run in pieces side by side, seeded from summaries.  Several pieces, a
    short last piece, summaries in parts, states in and out, columns below the tile's; against the oracle, and bit for bit the same
    whether the forward kept its states or the backward walks them again."""
    gen = torch.Generator().manual_seed(T + h)
    def randn(*s):
        return torch.randn(*s, generator=gen)
    bf = torch.bfloat16
    inp = {"x": randn(b, T, h, p).to(bf), "dt": torch.nn.functional.softplus(0.5 * randn(b, T, h) - 3.9).clamp(1e-3, 0.1),
           "A_head": -torch.exp(torch.rand(h, generator=gen) * 2.77 - 2.0), "B": (randn(b, T, g, n) / n ** 0.5).to(bf),
           "C": (randn(b, T, g, n) / n ** 0.5).to(bf), "D": randn(h), "dy": randn(b, T, h, p).to(bf)}
    init, dfinal = randn(b, h, p, n) * 0.5, randn(b, h, p, n)
    got = mamba2_gpu(pkg, inp, chunk, init, dfinal)
    want = oracle.mamba2_fwd_bwd(inp, chunk, torch.float32, init.unsqueeze(1), dfinal)
    errs = {k: rel_err(got[k], want[k].reshape(got[k].shape)) for k in got}
    bad = {k: v for k, v in errs.items() if not v < TOL_BF16}
    assert not bad, errs
    pkg.set_save_states(False)
    try:
        redone = mamba2_gpu(pkg, inp, chunk, init, dfinal)
    finally:
        pkg.set_save_states(True)
    for k in got:
        assert torch.equal(got[k], redone[k]), k


def test_mamba3_variant_takes_fp32_angles_with_bf16_tensors(pkg, cabi, oracle):
    """Angles given in fp32 (the reference's fp32 dt * theta product) are summed at that precision although x, B and C
    are bf16; their gradient comes back in fp32."""
    cfg = pkg.shrink(pkg.CONFIGS[3], 1, 512)
    inp = pkg.make_inputs(cfg)
    g = torch.Generator().manual_seed(3)
    inp["raw_angles"] = (torch.rand(inp["raw_angles"].shape, generator=g) * 2 - 1) * 0.37   # not bf16-representable
    names = ("x", "dt", "A_head", "B", "C", "D", "raw_angles", "lam")
    lv = {k: inp[k].to(DEV).requires_grad_(True) for k in names}
    y = pkg.ssd_mamba3(*[lv[k] for k in names], cfg.chunk)
    grads = torch.autograd.grad([y], list(lv.values()), [inp["dy"].to(DEV)])
    torch.cuda.synchronize()
    assert grads[6].dtype == torch.float32
    ol = {k: inp[k].float().requires_grad_(True) for k in names}
    yo = oracle.mamba3_operator(*[ol[k] for k in names], cfg.chunk)
    go = torch.autograd.grad([yo], list(ol.values()), [inp["dy"].float()])
    errs = {"y": rel_err(y, yo)}
    for k, a, b in zip(names, grads, go):
        errs["d" + k] = rel_err(a, b)
    bad = {k: v for k, v in errs.items() if not v < TOL_BF16}
    assert not bad, errs


@pytest.mark.parametrize("dtype,tol", [("fp32", TOL_FP32), ("bf16", TOL_BF16)])
def test_mamba3_variant(pkg, cabi, oracle, dtype, tol):
    """Rotary state angles + trapezoidal two-term form (config 3 per-token shape, reduced batch / sequence)
    against the oracle's two-call composition under plain autograd, all gradients including d raw_angles, d lam."""
    cfg = replace(pkg.shrink(pkg.CONFIGS[3], 1, 256), dtype=dtype)
    inp = pkg.make_inputs(cfg)
    names = ("x", "dt", "A_head", "B", "C", "D", "raw_angles", "lam")
    lv = {k: inp[k].to(DEV).requires_grad_(True) for k in names}
    y = pkg.ssd_mamba3(*[lv[k] for k in names], cfg.chunk)
    grads = torch.autograd.grad([y], list(lv.values()), [inp["dy"].to(DEV)])
    torch.cuda.synchronize()
    ol = {k: inp[k].float().requires_grad_(True) for k in names}
    yo = oracle.mamba3_operator(*[ol[k] for k in names], cfg.chunk)
    go = torch.autograd.grad([yo], list(ol.values()), [inp["dy"].float()])
    errs = {"y": rel_err(y, yo)}
    for k, a, b in zip(names, grads, go):
        errs["d" + k] = rel_err(a, b)
    bad = {k: v for k, v in errs.items() if not v < tol}
    assert not bad, errs


@pytest.mark.parametrize("T,h,g,n,chunk,ang32,shift", [(64, 1, 1, 40, 64, False, 0), (128, 4, 4, 128, 128, False, 0), (448, 5, 1, 64, 64, True, 0),
                                                       (1120, 12, 2, 104, 32, False, 1), (160, 600, 1, 64, 32, False, 0),
                                                       (192, 3, 1, 42, 64, False, 0), (256, 2, 1, 10, 128, True, 0)])
def test_mamba3_angles_edges(pkg, cabi, oracle, T, h, g, n, chunk, ang32, shift):
    """The running sum of the angles where it can go wrong: one block of positions and several, a last one that is not full,
    columns that do not fill the blocks, angles in fp32 and at an odd address (copied before the kernels see them), enough columns
    for the one-pass reverse sum, state columns that are no whole vectors.
    Against the oracle's two-call composition."""
    gen = torch.Generator().manual_seed(T + h)
    def randn(*s):
        return torch.randn(*s, generator=gen)
    bf = torch.bfloat16
    inp = {"x": randn(2, T, h, 64).to(bf), "dt": torch.nn.functional.softplus(0.5 * randn(2, T, h) - 3.9).clamp(1e-3, 0.1),
           "A_head": -torch.exp(torch.rand(h, generator=gen) * 2.77), "B": (randn(2, T, g, n) / n ** 0.5).to(bf),
           "C": (randn(2, T, g, n) / n ** 0.5).to(bf), "D": randn(h),
           "raw_angles": (torch.pi * (2 * torch.rand(2, T, h, n // 2, generator=gen) - 1)).to(torch.float32 if ang32 else bf),
           "lam": torch.sigmoid(randn(2, T, h))}
    dy = randn(2, T, h, 64).to(bf)
    lv = {k: v.to(DEV).requires_grad_(True) for k, v in inp.items()}
    if shift:
        raw = torch.empty(inp["raw_angles"].numel() + shift, dtype=bf, device=DEV)[shift:].view(inp["raw_angles"].shape)
        lv["raw_angles"] = raw.copy_(inp["raw_angles"]).requires_grad_(True)
    y = pkg.ssd_mamba3(*lv.values(), chunk)
    grads = torch.autograd.grad([y], list(lv.values()), [dy.to(DEV)])
    torch.cuda.synchronize()
    assert grads[6].dtype == inp["raw_angles"].dtype
    ol = {k: v.float().requires_grad_(True) for k, v in inp.items()}
    yo = oracle.mamba3_operator(*ol.values(), chunk)
    go = torch.autograd.grad([yo], list(ol.values()), [dy.float()])
    errs = {"y": rel_err(y, yo)}
    errs.update({"d" + k: rel_err(a, b) for k, a, b in zip(inp, grads, go)})
    bad = {k: v for k, v in errs.items() if not v < TOL_BF16}
    assert not bad, errs


@pytest.mark.parametrize("T,h,n,b", [(300, 3, 24, 2), (1120, 40, 64, 9), (129, 5, 8, 1)])
@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
def test_mamba3_angle_sums_do_not_depend_on_the_route(pkg, cabi, T, h, n, b, dtype):
    """The cumulative angles and the rotated B and C, from kernels that need aligned angles and from those that take any address:
    the sums are taken in one order, so the bits are the same.  Blocks of whole segments (the second shape) and of 32 positions."""
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    gen = torch.Generator(device=DEV).manual_seed(T)
    dt_ = torch.float32 if dtype == "fp32" else torch.bfloat16
    g = 1
    B, C = (torch.randn(b, T, g, n, generator=gen, device=DEV).to(dt_) for _ in range(2))
    ang = (torch.randn(b, T, h, n // 2, generator=gen, device=DEV)).to(dt_)
    shifted = torch.empty(ang.numel() + 1, dtype=dt_, device=DEV)[1:].view(ang.shape).copy_(ang)
    assert shifted.data_ptr() % 16
    dt, lam = torch.rand(b, T, h, generator=gen, device=DEV), torch.rand(b, T, h, generator=gen, device=DEV)
    Ah = -torch.ones(h, device=DEV)
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.F32 if dtype == "fp32" else cabi.BF16, cabi.F32, cabi.PATH_AUTO, b, T, h, 64, n, g, T)
    res = []
    for a in (ang, shifted):
        f = {k: torch.empty(b, T, h, device=DEV) for k in ("dA", "w", "skip")}
        Br, Cr = torch.empty(b, T, h, n, dtype=dt_, device=DEV), torch.empty(b, T, h, n, dtype=dt_, device=DEV)
        sdot, cum = torch.empty(b, T, g, device=DEV), torch.empty(b, T, h, n // 2, device=DEV)
        seg = torch.empty(b * ((T + 127) // 128) * h * (n // 2), device=DEV)
        P = S._ptr
        cabi.check(lib.ssd_b200_m3_prologue_fwd(ctypes.byref(shape), P(B), P(dt), P(lam), P(Ah), P(B), P(C), P(a), shape.dtype, None, P(f["dA"]),
                                                P(Br), P(Cr), P(sdot), P(cum), P(seg), None, P(f["w"]), P(f["skip"]), S._stream(torch.device(DEV))))
        torch.cuda.synchronize()
        res.append((cum, Br, Cr))
    for x, y in zip(*res):
        assert torch.equal(x, y)
    want = -ang.double().cumsum(1)
    assert rel_err(res[0][0], want) < TOL_FP32


@pytest.mark.parametrize("h,chunk", [(3, 64), (9, 256), (17, 64), (24, 256), (33, 128)])
def test_cumulative_sums_in_blocks_of_eight_and_of_32_heads(pkg, cabi, h, chunk):
    """512 tiles in blocks of 32 heads (of eight where half of 32 would be none) against a batch entry alone, whose blocks have eight: the sums have the same bits, also
    where a chunk begins in an earlier tile, and the decay gradients agree (the walks are cut differently)."""
    b, T = 16, 4096
    gen = torch.Generator(device=DEV).manual_seed(h)
    x, B, C, dy = (torch.randn(b, T, *s, generator=gen, device=DEV).bfloat16() for s in ((h, 64), (1, 128), (1, 128), (h, 64)))
    B, C = B / 128 ** 0.5, C / 128 ** 0.5
    A = -0.2 * torch.rand(b, T, h, generator=gen, device=DEV)
    def run(part):
        lv = [t[part].contiguous().requires_grad_(True) for t in (x, A, B, C)]
        y, _, cache = pkg.fused_ssd_scan(*lv, chunk)
        again = pkg.fused_ssd_scan(*lv, chunk, None, cache)[0]  # from the given sums
        return cache["A_cumsum"], y, again, *torch.autograd.grad(y, lv, dy[part])[:2]
    whole = run(slice(None))
    for i in (0, b - 1):
        alone = run(slice(i, i + 1))
        assert torch.equal(alone[0], whole[0][i:i + 1])
        assert torch.equal(whole[1], whole[2]) or rel_err(whole[1], whole[2]) < TOL_BF16
        for u, v in zip(alone[1:], whole[1:]):
            assert rel_err(u, v[i:i + 1]) < TOL_BF16


@pytest.mark.parametrize("b,T,h,g,n", [(1, 1, 4, 1, 64), (2, 5, 64, 1, 64), (3, 37, 12, 1, 128), (2, 130, 24, 2, 64), (1, 300, 40, 1, 192), (16, 1100, 8, 2, 64),
                                       (1, 1201, 64, 8, 128), (2, 33, 6, 2, 64), (1, 40, 68, 1, 64)])
def test_mamba3_rotation_backward(pkg, cabi, b, T, h, g, n):
    """Gradients of the rotation on their own: heads in fours through the ring in shared memory (a warp, several blocks and part of one per position; one to
    sixteen positions a warp, sequences that end inside a block; up to 64 heads a group) and the kernel for everything else (the last two
    shapes, and all shapes with angles off the 16-byte boundary), against 64 bits.  Angle gradients are fp32 sums of eight products: 1e-5 of
    the largest; dB and dC end in bf16, half a unit in 2^-8 of the value."""
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    gen = torch.Generator(device=DEV).manual_seed(T + h)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    B, C, dBr, dCr = (randn(*s).bfloat16() for s in ((b, T, g, n), (b, T, g, n), (b, T, h, n), (b, T, h, n)))
    cum, dt, lam, dyx = 100.0 * randn(b, T, h, n // 2), torch.rand(b, T, h, generator=gen, device=DEV), torch.rand(b, T, h, generator=gen, device=DEV), randn(b, T, h)
    shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, b, T, h, 64, n, g, T)
    def heads(v):  # (b,T,g,n) per head, as complex pairs
        return torch.view_as_complex(v.double().view(b, T, g, n // 2, 2)).repeat_interleave(h // g, 2)
    turn = torch.polar(torch.ones_like(cum, dtype=torch.float64), cum.double())
    gb, gc = (torch.view_as_complex(v.double().view(b, T, h, n // 2, 2)) * turn.conj() for v in (dBr, dCr))
    want_dth = (heads(B).conj() * gb + heads(C).conj() * gc).imag
    u = torch.nn.functional.pad(((1 - lam) * dt).double()[:, 1:], (0, 0, 0, 1))
    ds = -(u * dyx.double()).view(b, T, g, h // g).sum(-1, keepdim=True)
    def group(v):
        return torch.view_as_real(v.view(b, T, g, h // g, n // 2).sum(3)).reshape(b, T, g, n)
    want_dB, want_dC = group(gb) + ds * C.double(), group(gc) + ds * B.double()
    P = S._ptr
    for shift in (0, 1):
        cum_ = torch.empty(cum.numel() + shift, device=DEV)[shift:].view(cum.shape).copy_(cum)
        dB, dC, dcum, dang = torch.empty_like(B), torch.empty_like(C), torch.empty_like(cum), torch.empty_like(cum)
        sdot, dw = torch.zeros(b, T, g, device=DEV), torch.zeros(b, T, h, device=DEV)
        seg = torch.empty(b * ((T + 127) // 128) * h * (n // 2), device=DEV)
        cabi.check(lib.ssd_b200_m3_prologue_bwd(ctypes.byref(shape), None, None, P(dt), P(lam), None, P(B), P(C), P(cum_), P(sdot), None, P(dBr), P(dCr), None,
                                                P(dw), P(dyx), P(dB), P(dC), P(dang), cabi.F32, P(dcum), P(seg), S._stream(torch.device(DEV))))
        torch.cuda.synchronize()
        assert rel_err(dcum, want_dth) < TOL_FP32
        for got, want in ((dB, want_dB), (dC, want_dC)):
            assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()
        assert rel_err(dang, -dcum.double().flip(1).cumsum(1).flip(1)) < TOL_FP32


@pytest.mark.parametrize("b,T,h,g,n", [(26, 1, 64, 8, 64), (52, 7, 16, 4, 64), (26, 65, 16, 4, 128), (25, 129, 16, 4, 64), (13, 257, 32, 4, 64), (13, 600, 8, 2, 64),
                                       (12, 300, 64, 8, 128), (16, 1100, 8, 2, 64)])
@pytest.mark.parametrize("ang32", [True, False])
def test_mamba3_rotation_backward_with_its_sum(pkg, cabi, b, T, h, g, n, ang32):
    """Rotation undone and angle gradients summed in one kernel, in clusters of one to eight blocks, groups of four and eight heads, lengths that end inside a
    run, half a segment and a cluster's band: the bits of the two steps on their own (with room for what lies between them), also of a
    batch entry alone; and those against 64 bits, as above."""
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    gen = torch.Generator(device=DEV).manual_seed(T)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    P = S._ptr
    B, C, dBr, dCr = (randn(*s).bfloat16() for s in ((b, T, g, n), (b, T, g, n), (b, T, h, n), (b, T, h, n)))
    cum, dt, lam, dyx = 30.0 * randn(b, T, h, n // 2), torch.rand(b, T, h, generator=gen, device=DEV), torch.rand(b, T, h, generator=gen, device=DEV), randn(b, T, h)
    def run(k, apart):
        ins = [t[:k].contiguous() for t in (dt, lam, B, C, cum, dBr, dCr, dyx)]
        shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, k, T, h, 64, n, g, T)
        if not apart:
            assert lib.ssd_b200_m3_dcum_ws_floats(ctypes.byref(shape), P(ins[2]), P(ins[3]), P(ins[4]), P(ins[5]), P(ins[6])) == 0
        dB, dC, dcum = torch.empty_like(ins[2]), torch.empty_like(ins[3]), torch.empty_like(ins[4]) if apart else None
        dang = torch.empty(k, T, h, n // 2, dtype=torch.float32 if ang32 else torch.bfloat16, device=DEV)
        sdot, dw, seg = torch.zeros(k, T, g, device=DEV), torch.zeros(k, T, h, device=DEV), torch.empty(k * ((T + 127) // 128) * h * (n // 2), device=DEV)
        cabi.check(lib.ssd_b200_m3_prologue_bwd(ctypes.byref(shape), None, None, P(ins[0]), P(ins[1]), None, P(ins[2]), P(ins[3]), P(ins[4]), P(sdot), None, P(ins[5]),
                                                P(ins[6]), None, P(dw), P(ins[7]), P(dB), P(dC), P(dang), cabi.F32 if ang32 else cabi.BF16,
                                                P(dcum) if apart else None, P(seg), S._stream(torch.device(DEV))))
        torch.cuda.synchronize()
        return dB, dC, dang, dcum
    one, two, alone = run(b, False), run(b, True), run(1, True)
    for u, v, w in zip(one[:3], two[:3], alone[:3]):
        assert torch.equal(u, v) and torch.equal(u[:1], w)
    want = -two[3].double().flip(1).cumsum(1).flip(1)
    assert ((one[2].double() - want).abs() <= (0.0 if ang32 else 2.0 ** -8) * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("T", [600, 128])
def test_mamba3_angle_gradient_does_not_depend_on_the_batch(pkg, cabi, T):
    """Many columns take the reverse sum of the angle gradients in one pass, few in two; the order of the sums, and so
    the bits, are the same (a running sum over the whole sequence would round more the longer it is)."""
    gen = torch.Generator(device=DEV).manual_seed(T)
    b, h, p, n = 10, 64, 8, 128  # 40,960 columns
    def rand(*s):
        return torch.rand(*s, generator=gen, device=DEV)
    lv = [rand(b, T, h, p) - 0.5, 0.05 * rand(b, T, h), -rand(h), rand(b, T, 1, n) - 0.5, rand(b, T, 1, n) - 0.5, rand(h), 6 * rand(b, T, h, n // 2) - 3,
          rand(b, T, h)]
    dy = rand(b, T, h, p) - 0.5
    def dang(k):
        part = [t[:k].clone().requires_grad_(True) if t.shape[0] == b else t.clone().requires_grad_(True) for t in lv]
        y = pkg.ssd_mamba3(*part, T // 8)
        return y.detach(), torch.autograd.grad([y], [part[6]], [dy[:k]])[0]
    (y0, d0), (y1, d1) = dang(b), dang(1)
    assert torch.equal(y0[:1], y1) and torch.equal(d0[:1], d1)


@pytest.mark.parametrize("T", [1, 7, 9, 55, 57, 129, 601])
@pytest.mark.parametrize("ang32", [True, False])
@pytest.mark.parametrize("h,n,b", [(19, 20, 200), (19, 10, 400)])
def test_mamba3_reverse_sum_at_its_edges(pkg, cabi, T, ang32, h, n, b):
    """The reverse sum of the angle gradients in one pass: lengths that are no multiple of the eight positions fetched together, fewer than the 56 fetched
    ahead, ends inside a segment; columns that fill part of a block; and an odd number of columns, which takes two passes.  The same bits as a
    batch entry alone, whose columns are too few for one pass, and fp32 sums of up to 601 terms against 64 bits (bf16: one rounding)."""
    import ctypes
    lib, S = cabi.load(), pkg.ssd_scan
    gen = torch.Generator(device=DEV).manual_seed(T)
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV)
    B, C, dBr, dCr = (randn(b, T, k, n).bfloat16() for k in (1, 1, h, h))
    cum, dt, lam, dyx = randn(b, T, h, n // 2), torch.rand(b, T, h, generator=gen, device=DEV), torch.rand(b, T, h, generator=gen, device=DEV), randn(b, T, h)
    P = S._ptr
    def run(k):
        ins = [t[:k].contiguous() for t in (dt, lam, B, C, cum, dBr, dCr, dyx)]
        shape = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_AUTO, k, T, h, 64, n, 1, T)
        dB, dC, dcum = torch.empty_like(ins[2]), torch.empty_like(ins[3]), torch.empty_like(ins[4])
        dang = torch.empty(k, T, h, n // 2, dtype=torch.float32 if ang32 else torch.bfloat16, device=DEV)
        sdot, dw, seg = torch.zeros(k, T, 1, device=DEV), torch.zeros(k, T, h, device=DEV), torch.empty(k * ((T + 127) // 128) * h * (n // 2), device=DEV)
        cabi.check(lib.ssd_b200_m3_prologue_bwd(ctypes.byref(shape), None, None, P(ins[0]), P(ins[1]), None, P(ins[2]), P(ins[3]), P(ins[4]), P(sdot), None, P(ins[5]),
                                                P(ins[6]), None, P(dw), P(ins[7]), P(dB), P(dC), P(dang), cabi.F32 if ang32 else cabi.BF16, P(dcum), P(seg),
                                                S._stream(torch.device(DEV))))
        torch.cuda.synchronize()
        return dcum, dang
    (dcum, dang), (_, alone) = run(b), run(1)
    assert torch.equal(dang[:1], alone)
    want = -dcum.double().flip(1).cumsum(1).flip(1)
    assert ((dang.double() - want).abs() <= (0.0 if ang32 else 2.0 ** -8) * want.abs() + 1e-5 * want.abs().max()).all()


def test_mamba3_against_reference_fixture(pkg, cabi):
    """The one-scan Mamba-3 form on the GPU against outputs of the reference's own two-call composition
    (tests/golden/m3_reference_block.npz: reference rotation convention, coefficients and scan), fp32."""
    g = load_golden("m3_reference_block.npz")
    t = {k: torch.as_tensor(v) for k, v in g.items() if k != "chunk"}
    names = ("x", "dt", "A_head", "B", "C", "D", "raw_angles", "lam")
    lv = {k: t[k].to(DEV).requires_grad_(True) for k in names}
    y = pkg.ssd_mamba3(*[lv[k] for k in names], int(g["chunk"]))
    gr = dict(zip(names, torch.autograd.grad([y], list(lv.values()), [t["dY"].to(DEV)])))
    torch.cuda.synchronize()
    errs = {"Y": rel_err(y, t["Y"])}
    for k, ref in (("x", "dx"), ("lam", "dlam"), ("B", "dB"), ("C", "dC"), ("raw_angles", "d_raw_angles")):
        errs[ref] = rel_err(gr[k], t[ref])
    bad = {k: v for k, v in errs.items() if not v < TOL_FP32}
    assert not bad, errs


def test_host_pipeline_matches_direct_call(pkg, cabi):
    """The host-buffer entry (micro-batches over three streams) returns what one call on device tensors returns."""
    cfg = pkg.shrink(pkg.CONFIGS[2], 4, 256)
    inp = pkg.make_inputs(cfg)
    pinned = {k: v.pin_memory() for k, v in inp.items()}
    out = pkg.HostPipeline.alloc_outputs(pinned)
    pipe = pkg.HostPipeline("cuda", micro_batches=2)
    for _ in range(2):  # twice: slot reuse across calls
        pipe.run(pinned, out, cfg.chunk)
    got = {k: v.clone() for k, v in out.items()}  # read by the CPU right after run() returned: no device synchronise
    want = mamba2_gpu(pkg, inp, cfg.chunk)
    for k in ("y", "dx", "ddt", "dB", "dC"):
        assert torch.equal(got[k], want[k]), k
    assert rel_err(got["dA_head"], want["dA_head"]) < 1e-5 and rel_err(got["dD"], want["dD"]) < 1e-5
    # the stream-ordered form: nothing may be read before the returned event has completed
    ev = pipe.run(pinned, out, cfg.chunk, wait=False)
    ev.synchronize()
    assert torch.equal(out["y"], want["y"])


@pytest.mark.parametrize("idx,batch,seqlen,slice_len", [(2, 1, 1024, 256), (2, 2, 512, 128), (0, 2, 512, 128)])
def test_sequence_streamer_is_exact_across_slices(pkg, cabi, idx, batch, seqlen, slice_len):
    """The sequence-sliced host runner (state carried from slice to slice, its gradient carried back) returns what
    one call over the whole sequence returns, within the rounding of one pass."""
    cfg = pkg.shrink(pkg.CONFIGS[idx], batch, seqlen)
    inp = pkg.make_inputs(cfg)
    pinned = {k: v.pin_memory() for k, v in inp.items()}
    out = pkg.HostPipeline.alloc_outputs(pinned)
    runner = pkg.SequenceStreamer("cuda", slice_len=slice_len)
    for _ in range(2):  # twice: slot reuse across calls
        runner.run(pinned, out, cfg.chunk)
    got = {k: v.clone() for k, v in out.items()}  # CPU read right after run() returned
    want = mamba2_gpu(pkg, inp, cfg.chunk)
    tol = TOL_BF16 if cfg.dtype == "bf16" else TOL_FP32
    errs = {k: rel_err(got[k], want[k]) for k in ("y", "dx", "ddt", "dB", "dC", "dA_head", "dD")}
    bad = {k: v for k, v in errs.items() if not v < tol}
    assert not bad, errs


@pytest.mark.parametrize("idx,batch,seqlen,tol", [(2, 2, 512, TOL_BF16), (1, 2, 256, TOL_BF16), (0, 2, 256, TOL_FP32)])
def test_scan_with_gated_norm_output_stage(pkg, cabi, oracle, idx, batch, seqlen, tol):
    """ssd_mamba2_gated = scan + the block's output stage norm(y) * silu(z) (src/mamba_base_engine.py:189-191): on the
    tensor-core path the norm takes its row statistic from the partial sums the forward walk leaves behind (config 2
    and 1 shapes); on the fp32 path it computes it itself.  Against the oracle scan followed by the eager norm."""
    cfg = pkg.shrink(pkg.CONFIGS[idx], batch, seqlen)
    inp = pkg.make_inputs(cfg)
    b, T, h, p = inp["x"].shape
    g = torch.Generator().manual_seed(123)
    z = torch.randn(b, T, h * p, generator=g).to(inp["x"].dtype)
    w = 1.0 + 0.1 * torch.randn(h * p, generator=g)
    dout = torch.randn(b, T, h, p, generator=g).to(inp["x"].dtype)
    names = ("x", "dt", "A_head", "B", "C", "D")
    lv = {k: inp[k].to(DEV).requires_grad_(True) for k in names}
    zl, wl = z.to(DEV).requires_grad_(True), w.to(DEV).requires_grad_(True)
    out, fs = pkg.ssd_mamba2_gated(lv["x"], lv["dt"], lv["A_head"], lv["B"], lv["C"], lv["D"], zl, wl, 1e-6, cfg.chunk)
    grads = torch.autograd.grad([out], list(lv.values()) + [zl, wl], [dout.to(DEV)])
    torch.cuda.synchronize()
    ol = {k: inp[k].float().requires_grad_(True) for k in names}
    zo, wo = z.float().requires_grad_(True), w.clone().requires_grad_(True)
    yo, fo = oracle.mamba2_operator(ol["x"], ol["dt"], ol["A_head"], ol["B"], ol["C"], ol["D"], cfg.chunk)
    yf = yo.reshape(b, T, h * p)
    oo = (yf * torch.rsqrt(yf.pow(2).mean(-1, keepdim=True) + 1e-6) * wo * torch.nn.functional.silu(zo)).reshape(b, T, h, p)
    go = torch.autograd.grad([oo], list(ol.values()) + [zo, wo], [dout.float()])
    errs = {"out": rel_err(out, oo), "final": rel_err(fs, fo)}
    for k, a, c in zip(list(names) + ["z", "w"], grads, go):
        errs["d" + k] = rel_err(a, c)
    bad = {k: v for k, v in errs.items() if not v < tol}
    assert not bad, errs
    # and equal to the two-call composition of this package (same kernels apart from where the statistic comes from)
    y2, _ = pkg.ssd_mamba2(lv["x"], lv["dt"], lv["A_head"], lv["B"], lv["C"], lv["D"], cfg.chunk)
    o2 = pkg.fused_gate_norm(y2.reshape(b, T, h * p), zl, wl, 1e-6).reshape(b, T, h, p)
    assert rel_err(out, o2) < (1e-2 if cfg.dtype == "bf16" else 1e-5)


@pytest.mark.parametrize("h", [2, 24, 128, 130])
def test_gated_norm_statistic_of_unrounded_values(pkg, cabi, h):
    """The norm's statistic is of the scan's fp32 values: y = 1.0038 at every position rounds to 1 in bf16, its statistic does not,
    and at silu(20) = 20 the two differ by a bf16 step (19.875 against 20).  Rows held in registers (up to 8192 columns) and not."""
    bf, T = torch.bfloat16, 256
    B = torch.zeros(1, T, 1, 128, dtype=bf, device=DEV)
    x, z = torch.ones(1, T, h, 64, dtype=bf, device=DEV), torch.full((1, T, h * 64), 20.0, dtype=bf, device=DEV)
    out, _ = pkg.ssd_mamba2_gated(x, torch.full((1, T, h), 0.01, device=DEV), torch.full((h,), -1.0, device=DEV), B, B,
                                  torch.full((h,), 1.0038, device=DEV), z, torch.ones(h * 64, device=DEV), 1e-6, 128)
    want = torch.nn.functional.silu(z.double()) * (1.0038 ** 2 + 1e-6) ** -0.5  # 19.924, no tie
    assert torch.equal(out.flatten(), want.to(bf).flatten())


def test_scaled_operator_form_matches_mamba2_form(pkg, cabi):
    """The scan's third calling form (log-decay a, input weight dt and skip coefficient all per position; what the
    one-scan Mamba-3 composition uses) against the Mamba-2 form with a = dt * A_head and skip = D on the same data:
    same y, dx, dB, dC, and  ddt = d weight + da * A_head,  dA_head = sum da * dt,  dD = sum dskip."""
    import ctypes
    S, lib, P = pkg.ssd_scan, cabi.load(), pkg.ssd_scan._ptr
    cfg = pkg.shrink(pkg.CONFIGS[2], 2, 512)
    inp = {k: v.to(DEV) for k, v in pkg.make_inputs(cfg).items()}
    want = mamba2_gpu(pkg, {k: v.cpu() for k, v in inp.items()}, cfg.chunk)
    b, T, h, p = inp["x"].shape
    a = (inp["dt"] * inp["A_head"]).contiguous()
    skip = inp["D"].expand(b, T, h).contiguous()
    y, final, cum, shape, states = S._run_fwd(inp["x"], a, inp["dt"], None, None, inp["B"], inp["C"], cfg.chunk, None, None,
                                             want_states=True, skip=skip)
    dx, dB, dC = (torch.empty_like(inp[k]) for k in ("x", "B", "C"))
    da, dw, dskip = (torch.empty(b, T, h, device=DEV) for _ in range(3))
    ws = S._workspace(lib, shape, cabi.PASS_BWD, dx.device)
    args = cabi.BwdArgs(shape, P(inp["x"]), P(a), P(inp["dt"]), None, None, P(inp["B"]), P(inp["C"]), None, P(cum), P(inp["dy"]), None, P(dx), P(dB), P(dC),
                        P(da), P(dw), None, None, None, 0, 0, P(ws), ws.numel(), P(states), P(skip), P(dskip))
    cabi.check(lib.ssd_b200_bwd(ctypes.byref(args), S._stream(dx.device)))
    torch.cuda.synchronize()
    got = {"y": y, "final_state": final, "dx": dx, "dB": dB, "dC": dC,
           "ddt": dw + da * inp["A_head"], "dA_head": (da * inp["dt"]).sum((0, 1)), "dD": dskip.sum((0, 1))}
    errs = {k: rel_err(got[k], want[k]) for k in got}
    bad = {k: v for k, v in errs.items() if not v < 1e-3}   # same kernels, same roundings up to the order of the sums
    assert not bad, errs


def test_unused_outputs_are_not_materialised(pkg, cabi):
    """The operators ask autograd not to build zero gradients for outputs the loss does not use: with only y used the
    backward runs without a final-state gradient (no seed for the reverse walk), with only the final state used it
    builds the zero dY itself.  Both must equal the calls with explicit zeros."""
    cfg = pkg.shrink(pkg.CONFIGS[2], 2, 512)
    inp = {k: v.to(DEV) for k, v in pkg.make_inputs(cfg).items()}
    names = ("x", "dt", "A_head", "B", "C", "D")

    def grads(use_y, use_final, explicit):
        lv = {k: inp[k].clone().requires_grad_(True) for k in names}
        y, fs = pkg.ssd_mamba2(*[lv[k] for k in names], cfg.chunk)
        gfs = torch.ones_like(fs) * 0.5
        if explicit:
            outs, gs = [y, fs], [inp["dy"] if use_y else torch.zeros_like(y), gfs if use_final else torch.zeros_like(fs)]
        else:
            outs, gs = ([y] if use_y else []) + ([fs] if use_final else []), ([inp["dy"]] if use_y else []) + ([gfs] if use_final else [])
        return torch.autograd.grad(outs, list(lv.values()), gs)

    for use_y, use_final in ((True, False), (False, True)):
        a, b = grads(use_y, use_final, False), grads(use_y, use_final, True)
        for name, u, v in zip(names, a, b):
            assert torch.equal(u, v), (use_y, use_final, name)
