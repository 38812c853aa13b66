"""GPU parity tests of the rotation and trapezoidal-coefficient operators against the oracle's eager
definitions (pinned bit-exactly to the reference's own, tests/golden/PINNING.txt).  Shapes, seeds' structure and
tolerances follow the reference's tests (tests/kernels/test_rope.py:51-260, tests/kernels/test_trapezoidal.py:
37-150): fp32 forward 1e-5 absolute, bf16 forward 1e-2 absolute and no worse than eager bf16, gradients 1e-3.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"

ROPE_SHAPES = [(2, 256, 8, 16), (4, 512, 8, 32), (1, 1024, 4, 8), (2, 128, 64, 128), (1, 64, 3, 6)]
TRAP_SHAPES = [(2, 256, 8), (4, 1024, 8), (1, 2048, 16), (16, 4096, 64), (3, 50, 24)]


def _rope_inputs(B, T, H, D, dtype, seed=0, ang_scale=2.0, per_head=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(B, T, H, D, generator=g, device=DEV, dtype=dtype)
    angles = torch.randn(B, T, H if per_head else 1, D // 2, generator=g, device=DEV, dtype=dtype) * ang_scale
    return x, angles


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("shape", ROPE_SHAPES)
def test_rope_forward_fp32(pkg, cabi, oracle, shape, per_head):
    x, angles = _rope_inputs(*shape, torch.float32, per_head=per_head)
    y = pkg.fused_rope(x, angles)
    assert y.shape == x.shape and y.dtype == x.dtype
    assert (y - oracle.apply_rope(x, angles)).abs().max().item() < 1e-5


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("shape", ROPE_SHAPES[:4])
def test_rope_forward_bf16(pkg, cabi, oracle, shape, per_head):
    B, T, H, D = shape
    g = torch.Generator(device=DEV).manual_seed(0)
    x_bf = (torch.randn(B, T, H, D, generator=g, device=DEV) * 0.5).bfloat16()
    a_bf = torch.randn(B, T, H if per_head else 1, D // 2, generator=g, device=DEV).bfloat16()
    y_oracle = oracle.apply_rope(x_bf.float(), a_bf.float())
    err_eager = (oracle.apply_rope(x_bf, a_bf).float() - y_oracle).abs().max().item()
    y = pkg.fused_rope(x_bf, a_bf)
    assert y.dtype == torch.bfloat16
    err = (y.float() - y_oracle).abs().max().item()
    assert err < 1e-2 and err <= err_eager + 1e-3, (err, err_eager)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("shape", ROPE_SHAPES)
def test_rope_backward_fp32(pkg, cabi, oracle, shape, per_head):
    x, angles = _rope_inputs(*shape, torch.float32, seed=42, per_head=per_head)
    g = torch.randn_like(x)
    xr, ar = x.clone().requires_grad_(True), angles.clone().requires_grad_(True)
    oracle.apply_rope(xr, ar).backward(g)
    xk, ak = x.clone().requires_grad_(True), angles.clone().requires_grad_(True)
    pkg.fused_rope(xk, ak).backward(g)
    assert ak.grad.shape == angles.shape
    assert (xk.grad - xr.grad).abs().max().item() < 1e-3
    # the broadcast case sums over heads: compare relative to the size of the sum
    scale = max(1.0, ar.grad.abs().max().item())
    assert (ak.grad - ar.grad).abs().max().item() < 1e-3 * scale


def test_rope_rejects_bad_inputs(pkg, cabi):
    x = torch.zeros(1, 4, 2, 6, device=DEV)
    with pytest.raises(AssertionError):
        pkg.fused_rope(x, torch.zeros(1, 4, 3, 3, device=DEV))      # neither 1 nor H heads
    with pytest.raises(AssertionError):
        pkg.fused_rope(torch.zeros(1, 4, 2, 5, device=DEV), torch.zeros(1, 4, 1, 2, device=DEV))  # odd last dim
    with pytest.raises(AssertionError):
        pkg.fused_rope(x.cpu(), torch.zeros(1, 4, 1, 3))            # CPU tensors


def _trap_inputs(B, T, H, dtype, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    dt_raw = (torch.randn(B, T, H, generator=g, device=DEV) * 0.5).to(dtype)
    lam_raw = (torch.randn(B, T, H, generator=g, device=DEV) * 0.5).to(dtype)
    dt_bias = (torch.randn(H, generator=g, device=DEV) * 0.1).to(dtype)
    A_log = (torch.randn(H, generator=g, device=DEV) * 0.1).to(dtype)
    return dt_raw, lam_raw, dt_bias, A_log


@pytest.mark.parametrize("shape", TRAP_SHAPES)
def test_trapezoidal_forward_fp32(pkg, cabi, oracle, shape):
    ins = _trap_inputs(*shape, torch.float32)
    outs = pkg.fused_trapezoidal(*ins)
    for got, ref in zip(outs, oracle.trapezoid_from_raw(*ins)):
        assert got.shape == ins[0].shape and got.dtype == torch.float32
        assert (got - ref).abs().max().item() < 1e-5


@pytest.mark.parametrize("shape", TRAP_SHAPES[:4])
def test_trapezoidal_forward_bf16(pkg, cabi, oracle, shape):
    ins = _trap_inputs(*shape, torch.bfloat16)
    outs = pkg.fused_trapezoidal(*ins)
    refs = oracle.trapezoid_from_raw(*[t.float() for t in ins])
    for got, ref in zip(outs, refs):
        assert got.dtype == torch.bfloat16
        assert (got.float() - ref).abs().max().item() < 1e-2


@pytest.mark.parametrize("shape", TRAP_SHAPES)
def test_trapezoidal_backward_fp32(pkg, cabi, oracle, shape):
    ins = _trap_inputs(*shape, torch.float32, seed=7)
    gs = [torch.randn_like(ins[0]) for _ in range(4)]
    lr = [t.clone().requires_grad_(True) for t in ins]
    gr = torch.autograd.grad(list(oracle.trapezoid_from_raw(*lr)), lr, gs)
    lk = [t.clone().requires_grad_(True) for t in ins]
    gk = torch.autograd.grad(list(pkg.fused_trapezoidal(*lk)), lk, gs)
    for name, a, b in zip(("d_dt_raw", "d_lam_raw", "d_dt_bias", "d_A_log"), gk, gr):
        scale = max(1.0, b.abs().max().item())   # the parameter gradients are sums over all rows
        assert (a - b).abs().max().item() < 1e-3 * scale, name
    # deterministic reductions
    gk2 = torch.autograd.grad(list(pkg.fused_trapezoidal(*lk)), lk, gs)
    assert all(torch.equal(a, b) for a, b in zip(gk, gk2))


def test_trapezoidal_rejects_bad_inputs(pkg, cabi):
    dt_raw = torch.zeros(2, 8, 4, device=DEV)
    with pytest.raises(AssertionError):
        pkg.fused_trapezoidal(dt_raw, torch.zeros(2, 8, 5, device=DEV), torch.zeros(4, device=DEV), torch.zeros(4, device=DEV))
    with pytest.raises(AssertionError):
        pkg.fused_trapezoidal(dt_raw, dt_raw, torch.zeros(3, device=DEV), torch.zeros(4, device=DEV))
    with pytest.raises(AssertionError):
        pkg.fused_trapezoidal(dt_raw.cpu(), dt_raw.cpu(), torch.zeros(4), torch.zeros(4))


NORM_SHAPES = [(2, 256, 128), (4, 512, 256), (1, 1024, 96), (2, 64, 4, 32), (1, 128, 8, 16), (2, 64, 4096), (3, 7, 50)]
EPS = 1e-6


def _eager_rmsnorm(x, w, eps=EPS):
    """The reference tests' eager definition (tests/kernels/test_rmsnorm.py:35-38)."""
    return torch.nn.functional.rms_norm(x, (x.shape[-1],), w.to(x.dtype), eps)


@pytest.mark.parametrize("shape", NORM_SHAPES)
def test_rmsnorm_forward_fp32(pkg, cabi, shape):
    torch.manual_seed(0)
    x = torch.randn(*shape, device=DEV)
    w = torch.randn(shape[-1], device=DEV) * 0.5 + 1.0
    y = pkg.fused_rmsnorm(x, w, EPS)
    assert y.shape == x.shape and y.dtype == x.dtype
    assert (y - _eager_rmsnorm(x, w)).abs().max().item() < 1e-5


@pytest.mark.parametrize("shape", NORM_SHAPES[:6])
def test_rmsnorm_forward_bf16(pkg, cabi, shape):
    torch.manual_seed(1)
    x = torch.randn(*shape, device=DEV).bfloat16()
    w = (torch.randn(shape[-1], device=DEV) * 0.5 + 1.0).bfloat16()
    y = pkg.fused_rmsnorm(x, w, EPS)
    assert y.dtype == torch.bfloat16
    assert (y.float() - _eager_rmsnorm(x.float(), w.float())).abs().max().item() < 1e-2 * 4  # |y| reaches ~4 here; bf16 ulp scales


@pytest.mark.parametrize("shape", NORM_SHAPES)
def test_rmsnorm_backward_fp32(pkg, cabi, shape):
    torch.manual_seed(3)
    x = torch.randn(*shape, device=DEV)
    w = torch.randn(shape[-1], device=DEV) * 0.5 + 1.0
    g = torch.randn(*shape, device=DEV)
    xr, wr = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    _eager_rmsnorm(xr, wr).backward(g)
    xk, wk = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    pkg.fused_rmsnorm(xk, wk, EPS).backward(g)
    assert (xk.grad - xr.grad).abs().max().item() < 1e-3
    assert (wk.grad - wr.grad).abs().max().item() < 1e-3 * max(1.0, wr.grad.abs().max().item())


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 5e-2)])
@pytest.mark.parametrize("shape", [(2, 128, 4096), (2, 64, 256), (1, 33, 96), (1, 1, 8), (3, 401, 1024), (1, 601, 1032), (1, 5, 2056),
                                   (1, 700, 8192), (1, 9, 8200)])
def test_gate_norm_matches_block_epilogue(pkg, cabi, shape, dtype, tol):
    """norm(y) * silu(z) as the block composes it (src/mamba_base_engine.py:189-191), forward and gradients."""
    torch.manual_seed(5)
    y = torch.randn(*shape, device=DEV).to(dtype)
    z = torch.randn(*shape, device=DEV).to(dtype)
    w = torch.randn(shape[-1], device=DEV) * 0.5 + 1.0
    g = torch.randn(*shape, device=DEV).to(dtype)
    lr = [t.float().clone().requires_grad_(True) for t in (y, z, w)]
    ref = _eager_rmsnorm(lr[0], lr[2]) * torch.nn.functional.silu(lr[1])
    gr = torch.autograd.grad([ref], lr, [g.float()])
    lk = [t.clone().requires_grad_(True) for t in (y, z, w)]
    out = pkg.fused_gate_norm(lk[0], lk[1], lk[2], EPS)
    gk = torch.autograd.grad([out], lk, [g])
    assert out.dtype == dtype
    assert (out.float() - ref).abs().max().item() < tol * max(1.0, ref.abs().max().item())
    gtol = 1e-3 if dtype == torch.float32 else 5e-2
    for name, a, b in zip(("dy", "dz", "dw"), gk, gr):
        assert (a.float() - b).abs().max().item() < gtol * max(1.0, b.abs().max().item()), name


def test_rmsnorm_module_swap(pkg, cabi):
    torch.manual_seed(6)
    ref = torch.nn.RMSNorm(128, eps=EPS).to(DEV)
    with torch.no_grad():
        ref.weight.copy_(torch.randn(128, device=DEV) * 0.5 + 1.0)
    mod = pkg.FusedRMSNormModule(128, EPS).to(DEV)
    with torch.no_grad():
        mod.weight.copy_(ref.weight)
    x = torch.randn(4, 64, 128, device=DEV)
    assert (mod(x) - ref(x)).abs().max().item() < 1e-5
    # three-argument apply, as the reference's module calls it, and its backward
    xk = x.clone().requires_grad_(True)
    pkg.FusedRMSNorm.apply(xk, mod.weight, EPS).sum().backward()
    assert xk.grad is not None and mod.weight.grad is not None


def _shifted(t):
    """The same values, starting one element behind a 16-byte boundary."""
    out = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)[1:t.numel() + 1].view(t.shape).copy_(t)
    assert out.data_ptr() % 16 and out.is_contiguous()
    return out


@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (1, 3, 5, 64), (2, 129, 3, 24), (1, 1000, 7, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rope_angles_per_head_as_they_lie_in_memory(pkg, cabi, oracle, shape, dtype):
    """Vectors that are no multiple of a block's 256, one vector in all, heads of three to sixteen vectors: values and gradients.  bf16 results are
    one rounding off the fp32 ones of the same inputs (2^-8 of the value at most), angle gradients fp32 products."""
    x, angles = _rope_inputs(*shape, dtype, seed=5, per_head=True)
    g = torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(6), device=DEV).to(dtype)
    xr, ar = x.double().requires_grad_(True), angles.double().requires_grad_(True)
    want = oracle.apply_rope(xr, ar)
    want.backward(g.double())
    xk, ak = x.clone().requires_grad_(True), angles.clone().requires_grad_(True)
    y = pkg.fused_rope(xk, ak)
    y.backward(g)
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    for got, ref in ((y, want), (xk.grad, xr.grad), (ak.grad, ar.grad)):
        own = 2.0 ** -8 if got.dtype == torch.bfloat16 else ulp if got is ak.grad and ak.dtype == torch.bfloat16 else 0.0
        assert ((got.double() - ref).abs() <= own * ref.abs() + 1e-5 * ref.abs().max()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("who", ["x", "angles", "dy"])
def test_rope_takes_any_address(pkg, cabi, dtype, who):
    """Tensors off the 16-byte boundaries of the vector accesses: same results (single-element accesses, same arithmetic)."""
    x, angles = _rope_inputs(2, 40, 3, 64, dtype, seed=3, per_head=True)
    dy = torch.randn_like(x)
    def run(*ts):
        lv = [t.detach().requires_grad_(True) for t in ts[:2]]
        y = pkg.fused_rope(*lv)
        return [y.detach()] + list(torch.autograd.grad([y], lv, [ts[2]]))
    want = run(x, angles, dy)
    got = run(*[_shifted(t) if n == who else t for n, t in zip(("x", "angles", "dy"), (x, angles, dy))])
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [256, 8200, 100])
@pytest.mark.parametrize("who", ["x", "z", "weight", "dy"])
def test_gate_norm_takes_any_address(pkg, cabi, dtype, D, who):
    """The gated norm with one tensor off the 16-byte boundaries: as aligned, up to the order of the sums over a row (fp32: a few
    1e-7 of the largest value; bf16: one step of the storage type)."""
    g = torch.Generator(device=DEV).manual_seed(D)
    t = {"x": torch.randn(3, 21, D, generator=g, device=DEV).to(dtype), "z": torch.randn(3, 21, D, generator=g, device=DEV).to(dtype),
         "weight": torch.randn(D, generator=g, device=DEV) * 0.5 + 1, "dy": torch.randn(3, 21, D, generator=g, device=DEV).to(dtype)}
    def run(t):
        lv = [t[k].detach().requires_grad_(True) for k in ("x", "z", "weight")]
        y = pkg.fused_gate_norm(*lv, EPS)
        return [y.detach()] + list(torch.autograd.grad([y], lv, [t["dy"]]))
    want = run(t)
    got = run({k: _shifted(v) if k == who else v for k, v in t.items()})
    tol = 2e-6 if dtype == torch.float32 else 2 ** -7
    for a, b in zip(got, want):
        assert float((a.float() - b.float()).abs().max()) <= tol * float(b.float().abs().max())


@pytest.mark.parametrize("D", [256, 8200])
def test_rmsnorm_backward_takes_any_workspace_address(pkg, cabi, D):
    """The scratch of ssd_b200_rmsnorm_bwd needs no more than the alignment of its floats."""
    S, lib, rows = pkg.ssd_scan, cabi.load(), 37
    g = torch.Generator(device=DEV).manual_seed(D)
    x, dy, w = torch.randn(rows, D, generator=g, device=DEV), torch.randn(rows, D, generator=g, device=DEV), torch.rand(D, generator=g, device=DEV) + 0.5
    rstd = torch.rsqrt(x.pow(2).mean(1) + EPS)
    n = int(lib.ssd_b200_rmsnorm_ws_floats(rows, D))
    res = []
    for off in (0, 1):
        ws, dx, dw = torch.full((n + 2,), float("nan"), device=DEV), torch.empty_like(x), torch.empty_like(w)
        cabi.check(lib.ssd_b200_rmsnorm_bwd(cabi.F32, rows, D, S._ptr(x), S._ptr(w), None, S._ptr(dy), S._ptr(rstd), S._ptr(dx), None, S._ptr(dw),
                                            S._ptr(ws[off:]), S._stream(torch.device(DEV))))
        torch.cuda.synchronize()
        assert torch.isnan(ws[n + off:]).all()
        res.append((dx, dw))
    for a, b in zip(*res):
        assert float((a - b).abs().max()) <= 2e-6 * float(b.abs().max())


def test_tensors_without_columns_are_refused(pkg, cabi):
    """An exception, not the end of the process (the number of rows is a quotient by the columns)."""
    e = torch.empty(2, 3, 0, device=DEV)
    w = torch.empty(0, device=DEV)
    for call in (lambda: pkg.fused_rmsnorm(e, w, EPS), lambda: pkg.fused_gate_norm(e, e, w, EPS), lambda: pkg.fused_trapezoidal(e, e, w, w)):
        with pytest.raises((ValueError, RuntimeError, ZeroDivisionError)):
            call()


def _norm_rows(pkg, M, D, dtype):
    gen = torch.Generator(device=DEV).manual_seed(D + M)
    x, dout = (torch.randn(M, D, generator=gen, device=DEV).to(dtype) for _ in range(2))
    z = (20.0 * torch.randn(M, D, generator=gen, device=DEV)).clamp(-60, 60).to(dtype)
    w = 1.0 + 0.1 * torch.randn(D, generator=gen, device=DEV)
    for gate in (z, None):
        lv = [t.clone().requires_grad_(True) for t in ((x, gate, w) if gate is not None else (x, w))]
        out = pkg.fused_gate_norm(*lv, 1e-6) if gate is not None else pkg.fused_rmsnorm(*lv, 1e-6)
        got = torch.autograd.grad(out, lv, dout)
        ref = [t.detach().double().requires_grad_(True) for t in lv]
        y = ref[0] * torch.rsqrt(ref[0].square().mean(-1, keepdim=True) + 1e-6) * ref[-1]
        want = torch.autograd.grad(y * torch.nn.functional.silu(ref[1]) if gate is not None else y, ref, dout.double())
        for a, b in zip(got, want):
            ulp = 2.0 ** -8 if a.dtype == torch.bfloat16 else 0.0
            assert ((a.double() - b).abs() <= ulp * b.abs() + 1e-5 * b.abs().max()).all()


@pytest.mark.parametrize("M", [1, 3, 700])
@pytest.mark.parametrize("D,dtype", [(1032, torch.bfloat16), (2048, torch.bfloat16), (2056, torch.bfloat16), (4096, torch.bfloat16), (4104, torch.bfloat16),
                                     (8192, torch.bfloat16), (516, torch.float32), (1028, torch.float32), (4096, torch.float32)])
def test_norm_rows_of_a_block(pkg, cabi, M, D, dtype):
    """Backward of the norm, with and without a gate, where a row is a block's: fewer rows than are fetched ahead, one and many to a block, rows that do not
    fill the block's 256, 512 or 1024 vectors, gates from -60 to 60.  Against 64 bits; bf16 results one rounding (2^-8) off, sums over a row
    and over the rows fp32: 1e-5 of the largest value."""
    _norm_rows(pkg, M, D, dtype)


@pytest.mark.parametrize("M,D,dtype", [(9472, 2048, torch.bfloat16), (9471, 2048, torch.bfloat16), (9600, 1792, torch.bfloat16), (9600, 1784, torch.bfloat16),
                                       (4800, 4096, torch.bfloat16), (2400, 8192, torch.bfloat16), (700, 1024, torch.float32), (700, 2048, torch.float32),
                                       (700, 2044, torch.float32), (700, 1536, torch.float32)])
def test_norm_rows_with_and_without_the_ring(pkg, cabi, M, D, dtype):
    """The same on both sides of the lines between rows that come through the ring and rows that do not: bf16 without a gate from 16 rows a block and seven
    eighths of its vectors on, fp32 with a gate unless the row fills them."""
    _norm_rows(pkg, M, D, dtype)
