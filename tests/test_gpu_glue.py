"""GPU parity for the kernels either side of the cells (RMSNorm, output epilogue, SwiGLU gate, causal
depthwise convolution): through the C ABI against the CPU oracle and the fixtures made from the
reference's own modules.  fp32 1e-5 (elementwise math), bf16 2e-2 (max|a-b| / max|b|)."""
import numpy as np
import pytest
import torch

from conftest import relerr
from oracle import oracle as xo

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5
BF16_TOL = 2e-2


def dev(a, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def host(t):
    return t.detach().float().cpu().numpy()


def bf(a):
    return xo.bf16_round(np.asarray(a, np.float32))


@pytest.fixture(scope="module")
def ops():
    from xlstm_cuda import ops as _ops
    return _ops


# ---- RMSNorm ------------------------------------------------------------------------------
def test_rms_norm_golden(ops, golden):
    g = golden("norms")
    y = ops.rms_norm(dev(g["rms_x"]), dev(g["rms_w"]), 1e-6)
    np.testing.assert_allclose(host(y), g["rms_y"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("rows,cols", [(1, 4096), (5, 96), (3, 100), (7, 1023), (2, 8192), (2, 40000), (300, 4096)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rms_norm_shapes(ops, rows, cols, dtype):
    rng = np.random.default_rng(rows * 131 + cols)
    x = rng.standard_normal((rows, cols)).astype(np.float32) * 3.0
    w = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    if dtype == torch.bfloat16:
        x, w = bf(x), bf(w)
    ref = xo.rmsnorm(x, w, 1e-6)
    y = ops.rms_norm(dev(x, dtype), dev(w, dtype), 1e-6)
    assert y.dtype == dtype and y.shape == (rows, cols)
    assert relerr(host(y), ref) <= (FP32_TOL if dtype == torch.float32 else BF16_TOL)
    y0 = ops.rms_norm(dev(x, dtype), None, 1e-6)
    assert relerr(host(y0), xo.rmsnorm(x, None, 1e-6)) <= (FP32_TOL if dtype == torch.float32 else BF16_TOL)


@pytest.mark.parametrize("rows,cols", [(3, 4096), (300, 4096), (2000, 4096), (1500, 1024), (1300, 2048), (1200, 96),
                                       (1187, 4104)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_add_rms_norm_shapes(ops, rows, cols, dtype):
    """Residual add + RMSNorm: few rows (CTA per row) and many rows (the streamed kernel, >= 1184 rows), widths that
    fill the warp's vectors exactly and ones that do not.  The sum is rounded to the activation type, stored as
    the new residual stream, and the norm is taken of the rounded value."""
    rng = np.random.default_rng(rows * 7 + cols)
    x = rng.standard_normal((rows, cols)).astype(np.float32) * 2.0
    r = rng.standard_normal((rows, cols)).astype(np.float32) * 2.0
    w = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    if dtype == torch.bfloat16:
        x, r, w = bf(x), bf(r), bf(w)
    s_ref = x + r
    if dtype == torch.bfloat16:
        s_ref = bf(s_ref)
    y_ref = xo.rmsnorm(s_ref, w, 1e-6)
    s, y = ops.add_rms_norm(dev(x, dtype), dev(r, dtype), dev(w, dtype), 1e-6)
    np.testing.assert_array_equal(host(s), s_ref)                  # one rounding of an exact fp32 sum
    assert relerr(host(y), y_ref) <= (FP32_TOL if dtype == torch.float32 else BF16_TOL)
    s2, y2 = ops.add_rms_norm(dev(x, dtype), dev(r, dtype), None, 1e-6)
    assert torch.equal(s2, s)
    assert relerr(host(y2), xo.rmsnorm(s_ref, None, 1e-6)) <= (FP32_TOL if dtype == torch.float32 else BF16_TOL)


def test_rms_norm_empty_and_batched(ops):
    assert ops.rms_norm(torch.empty(0, 64, device="cuda"), None).shape == (0, 64)
    x = torch.randn(2, 3, 5, 64, device="cuda")
    y = ops.rms_norm(x, None, 1e-6)
    assert relerr(host(y), xo.rmsnorm(host(x), None, 1e-6)) <= FP32_TOL


def test_norm_cells_against_golden(golden):
    from xlstm_cuda.blocks import MultiHeadRMSNorm, RMSNormCell
    g = golden("norms")
    rn = RMSNormCell(96).cuda()
    rn.weight.data = dev(g["rms_w"])
    np.testing.assert_allclose(host(rn(dev(g["rms_x"]))), g["rms_y"], rtol=1e-5, atol=1e-6)
    mh = MultiHeadRMSNorm(4, 32).cuda()
    mh.weight.data = dev(g["mh_w"])
    np.testing.assert_allclose(host(mh(dev(g["mh_x"]))), g["mh_y"], rtol=1e-5, atol=1e-6)
    # permuted (non-contiguous) input, the layout the output cell hands over
    xp = dev(g["mh_x"]).permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    np.testing.assert_allclose(host(mh(xp)), g["mh_y"], rtol=1e-5, atol=1e-6)


# ---- output epilogue -------------------------------------------------------------------
def test_output_gate_golden(ops, golden):
    g = golden("glue_fp32")
    y = ops.mlstm_output_gate(dev(g["og_h"]), dev(g["og_pre"]), dev(g["og_w"]), float(g["og_eps"]))
    np.testing.assert_allclose(host(y), g["og_y"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("B,NH,S,dv", [(1, 8, 1, 512), (2, 4, 33, 64), (1, 2, 5, 1024), (3, 8, 130, 512), (2, 3, 7, 48),
                                       # more rows than warps in the grid: a warp walks several rows of its head
                                       (2, 8, 1500, 512), (2, 3, 2500, 48), (3, 5, 1111, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_output_gate_shapes_and_strides(ops, B, NH, S, dv, dtype):
    rng = np.random.default_rng(B * 7 + NH * 11 + S * 13 + dv)
    h = rng.standard_normal((B, NH, S, dv)).astype(np.float32) * 2.0
    og = rng.standard_normal((B, S, NH * dv)).astype(np.float32) * 2.0
    w = rng.uniform(0.5, 1.5, NH * dv).astype(np.float32)
    if dtype == torch.bfloat16:
        h, og, w = bf(h), bf(og), bf(w)
    ref = xo.mlstm_output_gate(h, og, w, 1e-6)
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    y = ops.mlstm_output_gate(dev(h, dtype), dev(og, dtype), dev(w, dtype), 1e-6)
    assert y.shape == (B, S, NH * dv) and relerr(host(y), ref) <= tol
    # h as a permuted view of a [B,S,NH,dv] buffer (the layout the fused all-gather produces)
    hp = dev(h, dtype).permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    assert not hp.is_contiguous() or S == 1 or NH == 1
    y2 = ops.mlstm_output_gate(hp, dev(og, dtype), dev(w, dtype), 1e-6)
    assert torch.equal(y, y2)
    y3 = ops.mlstm_output_gate(dev(h, dtype), dev(og, dtype), None, 1e-6)
    assert relerr(host(y3), xo.mlstm_output_gate(h, og, None, 1e-6)) <= tol


# ---- SwiGLU gate ----------------------------------------------------------------------
def test_swiglu_golden(ops, golden):
    g = golden("glue_fp32")
    y = ops.swiglu(dev(g["sw_g"]), dev(g["sw_u"]))
    np.testing.assert_allclose(host(y), g["sw_y"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("rows,cols", [(1, 10944), (4, 64), (3, 41), (257, 2048),
                                       (4100, 10944), (40000, 1000)])   # the last two: the streamed kernel
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_swiglu_dense_and_column_blocks(ops, rows, cols, dtype):
    rng = np.random.default_rng(rows + cols)
    gu = rng.standard_normal((rows, 2 * cols)).astype(np.float32) * 3.0
    if dtype == torch.bfloat16:
        gu = bf(gu)
    ref = xo.swiglu(gu[:, :cols], gu[:, cols:])
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    t = dev(gu, dtype)
    y_blocks = ops.swiglu(t[:, :cols], t[:, cols:])              # the two halves of one GEMM output
    y_dense = ops.swiglu(t[:, :cols].contiguous(), t[:, cols:].contiguous())
    assert y_blocks.is_contiguous() and y_blocks.shape == (rows, cols)
    assert relerr(host(y_blocks), ref) <= tol and torch.equal(y_blocks, y_dense)


# ---- causal depthwise convolution -------------------------------------------------------
def test_causal_conv_golden(ops, golden):
    g = golden("glue_fp32")
    x, w, b = dev(g["conv_x"]), dev(g["conv_w"]), dev(g["conv_b"])
    np.testing.assert_allclose(host(ops.causal_conv1d(x, w, b)), g["conv_y"], rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(host(ops.causal_conv1d(x, w, b, silu=True)), g["conv_y_silu"], rtol=1e-5, atol=1e-6)
    # [C,1,K] weight of nn.Conv1d is accepted as is
    np.testing.assert_allclose(host(ops.causal_conv1d(x, w.view(-1, 1, 4), b)), g["conv_y"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("B,S,C,K", [(1, 1, 64, 4), (2, 2, 64, 4), (2, 16, 128, 4), (3, 17, 1024, 4), (2, 100, 40, 2),
                                     (1, 33, 256, 8), (2, 5, 64, 1),
                                     # long runs per thread: the shared-memory ring is refilled (32 / 64 / 128 tokens)
                                     (4, 4099, 1040, 4), (16, 4096, 1024, 4), (32, 4100, 1024, 3), (24, 2051, 512, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_causal_conv_shapes_and_state(ops, B, S, C, K, dtype):
    rng = np.random.default_rng(B + 3 * S + 5 * C + 7 * K)
    x = rng.standard_normal((B, S, C)).astype(np.float32)
    w = (rng.standard_normal((C, K)) * 0.5).astype(np.float32)
    b = (rng.standard_normal(C) * 0.1).astype(np.float32)
    st = rng.standard_normal((B, K - 1, C)).astype(np.float32)
    if dtype == torch.bfloat16:
        x, w, b, st = bf(x), bf(w), bf(b), bf(st)
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    ref, ref_st = xo.causal_conv1d(x, w, b, state=st, silu=True, return_state=True)
    y, st1 = ops.causal_conv1d(dev(x, dtype), dev(w, dtype), dev(b, dtype), silu=True, state=dev(st, dtype),
                               return_state=True)
    assert relerr(host(y), ref) <= tol
    if K > 1:
        np.testing.assert_array_equal(host(st1), ref_st)          # the state is a copy of inputs: exact
    y0 = ops.causal_conv1d(dev(x, dtype), dev(w, dtype), None)    # no bias, zero history, no activation
    assert relerr(host(y0), xo.causal_conv1d(x, w, None)) <= tol


def test_causal_conv_token_by_token_equals_sequence(ops):
    rng = np.random.default_rng(5)
    B, S, C, K = 2, 40, 128, 4
    x = dev(rng.standard_normal((B, S, C)).astype(np.float32))
    w = dev((rng.standard_normal((C, K)) * 0.5).astype(np.float32))
    b = dev((rng.standard_normal(C) * 0.1).astype(np.float32))
    full = ops.causal_conv1d(x, w, b, silu=True)
    st, outs = None, []
    for t in range(S):
        y, st = ops.causal_conv1d(x[:, t:t + 1], w, b, silu=True, state=st, return_state=True)
        outs.append(y)
    assert torch.equal(torch.cat(outs, 1), full)
    y1, st = ops.causal_conv1d(x[:, :23], w, b, silu=True, return_state=True)
    y2 = ops.causal_conv1d(x[:, 23:], w, b, silu=True, state=st)
    assert torch.equal(torch.cat([y1, y2], 1), full)


def test_glue_rejects_cpu_tensors(ops):
    with pytest.raises(RuntimeError):
        ops.rms_norm(torch.zeros(2, 8), None)
    with pytest.raises(RuntimeError):
        ops.swiglu(torch.zeros(2, 8), torch.zeros(2, 8))


# ---- single-token Linear (weight-streaming pass with folded norm / residual / SwiGLU) ----------
@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (1, 12304, 4096), (2, 4096, 10944), (4, 264, 520), (3, 33, 4096),
                                   (4, 300, 10944), (1, 500, 16), (2, 1000, 2056)])
def test_linear_token_plain_bias_residual(ops, M, N, K):
    rng = np.random.default_rng(M * 7 + N + K)
    x = bf(rng.standard_normal((M, K)).astype(np.float32))
    W = bf((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
    b = bf((rng.standard_normal(N) * 0.1).astype(np.float32))
    r = bf(rng.standard_normal((M, N)).astype(np.float32))
    t = torch.bfloat16
    ref = xo.linear(x, W, b)
    y = ops.linear_token(dev(W, t), dev(x, t), bias=dev(b, t))
    assert y.shape == (M, N) and relerr(host(y), ref) <= BF16_TOL
    y0 = ops.linear_token(dev(W, t), dev(x, t))
    assert relerr(host(y0), xo.linear(x, W)) <= BF16_TOL
    yr = ops.linear_token(dev(W, t), dev(x, t), bias=dev(b, t), residual=dev(r, t))
    assert relerr(host(yr), bf(ref) + r) <= BF16_TOL


@pytest.mark.parametrize("M,F,K", [(1, 10944, 4096), (2, 320, 256), (4, 64, 4096)])
def test_linear_token_norm_and_swiglu(ops, M, F, K):
    rng = np.random.default_rng(M + F + K)
    x = bf(rng.standard_normal((M, K)).astype(np.float32) * 3.0)
    nw = bf(rng.uniform(0.5, 1.5, K).astype(np.float32))
    W = bf((rng.standard_normal((2 * F, K)) * 0.05).astype(np.float32))
    t = torch.bfloat16
    xn = bf(xo.rmsnorm(x, nw, 1e-6))
    # norm folded into the projection
    y = ops.linear_token(dev(W[:F], t), dev(x, t), norm_weight=dev(nw, t), norm_eps=1e-6)
    assert relerr(host(y), xo.linear(xn, W[:F])) <= BF16_TOL
    # ... and the SwiGLU gate on the two stacked up projections
    g, u = bf(xo.linear(xn, W[:F])), bf(xo.linear(xn, W[F:]))
    act = ops.linear_token(dev(W, t), dev(x, t), norm_weight=dev(nw, t), norm_eps=1e-6, swiglu_pair=True)
    assert act.shape == (M, F) and relerr(host(act), xo.swiglu(g, u)) <= BF16_TOL
    # equals the separate kernels up to bf16 rounding of the same intermediate values
    sep = ops.swiglu(*torch.nn.functional.linear(ops.rms_norm(dev(x, t), dev(nw, t), 1e-6), dev(W, t)).split(F, dim=-1))
    assert relerr(host(act), host(sep)) <= BF16_TOL


@pytest.mark.parametrize("rows,cols,dtype", [(1, 8, torch.bfloat16), (33, 1368, torch.bfloat16), (5, 4, torch.float32), (700, 344, torch.float32)])
def test_geglu_matches_separate_ops(ops, rows, cols, dtype):
    """One 16-byte vector, odd row counts; bf16 equal up to one ulp of the product (erff here and in torch agree to an ulp)."""
    torch.manual_seed(rows)
    x = (torch.randn(rows, 2 * cols, device="cuda") * 3).to(dtype)
    ref = x[:, :cols] * torch.nn.functional.gelu(x[:, cols:])
    assert relerr(host(ops.geglu(x)), host(ref)) <= (2.0 ** -7 if dtype == torch.bfloat16 else 1e-6)


@pytest.mark.parametrize("rows,groups,cols", [(1, 1, 8), (3, 4, 1024), (37, 1, 1368), (2, 1, 8192), (1500, 1, 4096), (700, 2, 2056), (5, 1, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_layer_norm(ops, rows, groups, cols, dtype):
    """A vector a row, the widths at which a lane holds another number of vectors, a warp and a CTA a row; rows far from zero
    mean.  fp32: sums of up to 8192 terms, bf16: one rounding (2^-8 of the value) of a result within 1e-5 of the exact one."""
    torch.manual_seed(rows + cols)
    x = (torch.randn(rows, groups * cols, device="cuda") * 2 + 5).to(dtype)
    w, b = (torch.randn(groups * cols, device="cuda").to(dtype) for _ in range(2))
    assert ops.layer_norm_takes(x, w, b, groups)
    y = ops.layer_norm(x, w, b, 1e-6, groups).double().cpu()
    x64, w64, b64 = (t.double().cpu() for t in (x, w, b))
    ref = torch.nn.functional.group_norm(x64, groups, w64, b64, 1e-6)
    off = (y - ref).abs()
    assert bool((off <= (2.0 ** -8 * ref.abs() if dtype == torch.bfloat16 else 0) + 1e-5 * (1 + w64.abs())).all()), float(off.max())


def test_layer_norm_takes_what_the_kernel_does(ops):
    x, w = torch.zeros(4, 64, device="cuda"), torch.zeros(64, device="cuda")
    assert not ops.layer_norm_takes(x, w.bfloat16(), w, 1) and not ops.layer_norm_takes(x, None, w, 1)
    assert not ops.layer_norm_takes(x.t(), w, w, 1) and not ops.layer_norm_takes(x, w, w, 32)          # 8-byte blocks
    assert not ops.layer_norm_takes(torch.zeros(257, device="cuda")[1:].view(4, 64), w, w, 1)          # odd offset
    with pytest.raises(Exception):
        ops.layer_norm(torch.zeros(4, 6, device="cuda"), torch.zeros(6, device="cuda"), torch.zeros(6, device="cuda"))


def test_norms_of_the_slstm_blocks_are_their_modules(ops, monkeypatch):
    """The fused norm stands in for the module only where nobody can tell: hooks, gradients, autocast and function transforms
    see the module."""
    from xlstm_cuda.blocks.slstm import sLSTMOutputCell
    from xlstm_cuda.blocks import slstm as blocks_slstm
    monkeypatch.setattr(blocks_slstm, "NORM_MIN_NUMEL", 1)
    torch.manual_seed(0)
    cell = sLSTMOutputCell(256, 4, 64).cuda()
    with torch.no_grad():
        cell.group_norm.weight.normal_()
        cell.group_norm.bias.normal_()
    h = torch.randn(2, 9, 4, 64, device="cuda")
    with torch.inference_mode():
        fused = cell(h)
        seen = []
        handle = cell.group_norm.register_forward_hook(lambda *a: seen.append(1))
        plain = cell(h)
        handle.remove()
        assert seen and relerr(host(fused), host(plain)) <= 1e-5
    h2 = h.clone().requires_grad_()
    cell(h2).sum().backward()
    assert h2.grad is not None and cell.group_norm.weight.grad is not None
    with torch.no_grad():
        _, tangent = torch.func.jvp(cell, (h,), (torch.ones_like(h),))
        assert torch.isfinite(tangent).all()
        assert relerr(host(torch.func.vmap(cell)(torch.stack([h, h]))[1]), host(plain)) <= 1e-5


def test_slstm_cells_under_modes_go_through_the_modules(ops, monkeypatch):
    """A graph of the output cell made by make_fx computes with its own input, and a mode that listens sees the norm and the gate
    projections; a default device is no such mode."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode

    from xlstm_cuda.blocks import slstm as blocks_slstm
    monkeypatch.setattr(blocks_slstm, "NORM_MIN_NUMEL", 1)
    torch.manual_seed(4)

    class Log(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func._opname)
            return func(*args, **(kwargs or {}))
    seen = []
    cell, pc = blocks_slstm.sLSTMOutputCell(64, 4, 16).cuda(), blocks_slstm.sLSTMProjectionCell(64, 4, 16).cuda().bfloat16()
    h, h2 = torch.randn(2, 9, 4, 16, device="cuda"), torch.randn(2, 9, 4, 16, device="cuda")
    with torch.no_grad():
        assert relerr(host(make_fx(cell)(h)(h2)), host(cell(h2))) <= 1e-5
        with Log():
            cell(h)
            pc.gates_and_z(h.flatten(2).bfloat16())
        assert "native_group_norm" in seen and sum(name in ("mm", "addmm") for name in seen) == 1 + 4
        seen.clear()
        with torch.device("cuda"):
            monkeypatch.setattr(torch.nn.GroupNorm, "forward", None)     # not called: the fused launch is taken
            cell(h)


def test_ensembles_of_slstm_cells_go_through_the_modules(ops, monkeypatch):
    """Stacked weights of an ensemble under vmap, an input that is shared: the weights have no memory of their own to hand to a
    kernel, so the cells call their modules, as for a member at a time."""
    from xlstm_cuda.blocks import slstm as blocks_slstm
    monkeypatch.setattr(blocks_slstm, "NORM_MIN_NUMEL", 1)

    class Gates(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.cell = blocks_slstm.sLSTMProjectionCell(64, 4, 16, gate_soft_cap=None)

        def forward(self, x):
            return torch.cat([t.flatten(2) for t in self.cell.gates_and_z(x)], -1)
    torch.manual_seed(3)
    with torch.no_grad():
        for make, x, part in ((lambda: blocks_slstm.sLSTMOutputCell(64, 4, 16), torch.randn(2, 9, 4, 16, device="cuda"), "group_norm"),
                              (Gates, torch.randn(2, 9, 64, device="cuda"), "gate_proj")):
            cells = [make().cuda().bfloat16() for _ in range(3)]
            x = x.bfloat16()
            base = dict(cells[0].named_parameters())
            members = [{k: (torch.randn_like(v) if part in k else v) for k, v in base.items()} for _ in cells]
            stacked = {k: torch.stack([m[k] for m in members]) for k in base if part in k}
            call = lambda p: torch.func.functional_call(cells[0], {**base, **p}, (x,))
            y = torch.func.vmap(call)(stacked)
            for n, m in enumerate(members):
                assert relerr(host(y[n]), host(call(m))) <= BF16_TOL


@pytest.mark.parametrize("B,S,C,NH", [(1, 1, 32, 4), (2, 3, 64, 1), (1, 16, 1024, 4), (3, 17, 416, 2), (1, 77, 4096, 4),
                                      (4, 1801, 128, 3), (2, 3555, 64, 4)])
@pytest.mark.parametrize("cap,bias", [(15.0, True), (None, False)])
def test_slstm_gates(ops, B, S, C, NH, cap, bias):
    """Both tile sizes, tokens around a tile's edge and before the first one, fewer channel blocks than warps.  Against float64
    on the convolution kernel's own (rounded) result: the sums differ by fp32 summation order, 2^-8 is the one rounding, doubled
    where the value rounded before the cap sits at a boundary."""
    torch.manual_seed(S + C)
    t = torch.bfloat16
    x = torch.randn(B, S, C, device="cuda").to(t)
    cw, cb = torch.randn(C, 1, 4, device="cuda").to(t) * 0.5, torch.randn(C, device="cuda").to(t) if bias else None
    w = [(torch.randn(NH, C, device="cuda") * 2 / C ** 0.5).to(t) for _ in range(3)]
    b = [torch.randn(NH, device="cuda").to(t) for _ in range(3)]
    assert ops.slstm_gates_takes(x, cw, cb, w, b)
    got = ops.slstm_gates(x, cw, cb, w, b, cap)
    xc = ops.causal_conv1d(x, cw, cb, silu=True)
    for k, src in enumerate((xc, xc, x)):
        ref = src.double().cpu() @ w[k].double().cpu().t() + b[k].double().cpu()
        if cap:
            ref = cap * torch.tanh(ref / cap)
        off = (got[k].double().cpu() - ref).abs()
        assert got[k].shape == (B, S, NH) and bool((off <= 2.0 ** -7 * ref.abs() + 2e-4).all()), (k, float(off.max()))


def test_slstm_projection_without_the_convolved_input(ops):
    """The neuron's path equals the projection cell's, and goes through the modules where they carry hooks."""
    from xlstm_cuda.blocks.slstm import sLSTMProjectionCell
    torch.manual_seed(1)
    pc = sLSTMProjectionCell(256, 4, 64).cuda().bfloat16()
    x = torch.randn(2, 70, 256, device="cuda").bfloat16()
    with torch.inference_mode():
        z, i, f, o, _ = pc(x)
        for a, b in zip(pc.gates_and_z(x), (z, i, f, o)):
            assert relerr(host(a), host(b)) <= BF16_TOL
        seen = []
        pc.fgate_proj.register_forward_hook(lambda *a: seen.append(1))
        pc.gates_and_z(x)
        assert seen


@pytest.mark.parametrize("M,N,K", [(16, 4096, 4096), (5, 33, 64), (9, 264, 10944), (16, 31, 32), (1, 1, 288), (12, 50, 2080)])
def test_linear_rows(ops, M, N, K):
    """Rows around the 8-row halves of the x operand, weight rows and k blocks around a CTA's and a warp's share."""
    rng = np.random.default_rng(M * 7 + N + K)
    x = bf(rng.standard_normal((M, K)).astype(np.float32))
    W = bf((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
    b = bf((rng.standard_normal(N) * 0.1).astype(np.float32))
    r = bf(rng.standard_normal((M, N)).astype(np.float32))
    t = torch.bfloat16
    ref = xo.linear(x, W, b)
    y = ops.linear_rows(dev(W, t), dev(x, t), bias=dev(b, t))
    assert y.shape == (M, N) and relerr(host(y), ref) <= BF16_TOL
    assert relerr(host(ops.linear_rows(dev(W, t), dev(x, t))), xo.linear(x, W)) <= BF16_TOL
    yr = ops.linear_rows(dev(W, t), dev(x, t), bias=dev(b, t), residual=dev(r, t))
    assert relerr(host(yr), bf(ref) + r) <= BF16_TOL
    W2 = bf((rng.standard_normal((2 * N, K)) * 0.05).astype(np.float32))
    act = ops.linear_rows(dev(W2, t), dev(x, t), swiglu_pair=True)
    assert act.shape == (M, N)
    assert relerr(host(act), xo.swiglu(bf(xo.linear(x, W2[:N])), bf(xo.linear(x, W2[N:])))) <= BF16_TOL


@pytest.mark.parametrize("M,N,K", [(16, 4736, 2048), (3, 4737, 2048), (16, 9472, 2048), (5, 9473, 2048), (7, 70, 1024), (16, 70, 1056)])
def test_linear_rows_forms(ops, M, N, K):
    """Both sides of the lines between a CTA a tile and CTAs that walk (148 and 296 tiles, rows of 1024), plain, as a pair and with a
    norm, against float64: fp32 sums of K products (within K 2^-24 of their absolute sum) and the bf16 roundings on the way."""
    torch.manual_seed(M + N + K)
    t = torch.bfloat16
    W, x = (torch.randn(N, K, device="cuda") * 0.05).to(t), torch.randn(M, K, device="cuda").to(t)
    W64, x64 = W.double(), x.double()
    ref = x64 @ W64.t()
    room = 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * (x64.abs() @ W64.abs().t())
    assert bool(((ops.linear_rows(W, x).double() - ref).abs() <= room).all())
    half = N // 2 * 2
    gate, up = (a.to(t).double() for a in ref[:, :half].split(half // 2, 1))
    pair = gate * torch.sigmoid(gate) * up
    got = ops.linear_rows(W[:half].contiguous(), x, swiglu_pair=True).double()
    assert float((got - pair).abs().max()) <= BF16_TOL * float(pair.abs().max())
    if M * (2 * K + 64) + 2 * K <= 49152:
        nw = torch.rand(K, device="cuda").to(t) + 0.5
        assert torch.equal(ops.linear_rows(W, x, norm_weight=nw), ops.linear_rows(W, ops.rms_norm(x, nw)))


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (2, 31, 32), (4, 5000, 4096), (3, 17, 1056), (16, 4800, 96), (5, 9600, 2080)])
def test_linear_rows_with_norm(ops, M, N, K):
    """One row and sixteen, fewer and more tiles than CTAs, k blocks around a warp's share: the norm in front equals its own
    launch bit for bit, so the Linear does too."""
    torch.manual_seed(M * 7 + N + K)
    t = torch.bfloat16
    x, nw = torch.randn(M, K, device="cuda").to(t) * 3, torch.rand(K, device="cuda").to(t) + 0.5
    W, b = (torch.randn(N, K, device="cuda") * 0.05).to(t), torch.randn(N, device="cuda").to(t)
    xn = ops.rms_norm(x, nw, 1e-6)
    assert torch.equal(ops.linear_rows(W, x, bias=b, norm_weight=nw, norm_eps=1e-6), ops.linear_rows(W, xn, bias=b))
    W2 = (torch.randn(2 * N, K, device="cuda") * 0.05).to(t)
    assert torch.equal(ops.linear_rows(W2, x, swiglu_pair=True, norm_weight=nw), ops.linear_rows(W2, xn, swiglu_pair=True))
    with pytest.raises(Exception):     # more rows than shared memory is given to
        ops.linear_rows(W[:, :1].expand(N, 4096).contiguous(), torch.zeros(8, 4096, device="cuda", dtype=t), norm_weight=nw[:1].expand(4096))
    with pytest.raises(Exception):
        ops.linear_rows(W, x, residual=torch.zeros(M, N, device="cuda", dtype=t), norm_weight=nw)


def test_linear_rows_with_norm_from_several_threads(ops):
    """Calls that need different amounts of shared memory, from threads that run beside one another: none is refused."""
    import threading
    from xlstm_cuda import _lib
    lib, t, failed = _lib.load(), torch.bfloat16, []

    def calls(M, K, N=16):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            W, x, nw, y = (torch.randn(s, device="cuda").to(t) for s in ((N, K), (M, K), (K,), (M, N)))
        args = (W.data_ptr(), x.data_ptr(), None, nw.data_ptr(), 1e-6, None, y.data_ptr(), M, N, K, 0, 0, _lib.BF16, stream.cuda_stream)
        failed.extend(rc for rc in (lib.xlstm_linear_rows_norm(*args) for _ in range(20000)) if rc)
        stream.synchronize()
    threads = [threading.Thread(target=calls, args=a) for a in ((1, 32), (16, 1408), (2, 32), (15, 1408))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed, (len(failed), failed[:3])


@pytest.mark.parametrize("K", [32, 64, 288, 1024])
def test_linear_rows_keeps_infinities(ops, K):
    """An infinite weight gives an infinite result in its row and none elsewhere, also in the last block of k."""
    t = torch.bfloat16
    torch.manual_seed(K)
    x = torch.rand(5, K, device="cuda").to(t) + 0.5
    W = torch.randn(40, K, device="cuda").to(t)
    W[7, K - 1], W[33, 0] = float("inf"), float("-inf")
    y = ops.linear_rows(W, x)
    assert torch.equal(torch.isinf(y), torch.isinf(x.float() @ W.float().T)) and not torch.isnan(y).any()


def test_linear_rows_reads_weights_written_just_before(ops):
    """A weight that the launch right before the call writes (an update in place; the dense copy that the call itself makes of a
    transposed one, also where the caller vouches for the weight it passes) is not read early."""
    t = torch.bfloat16
    torch.manual_seed(0)
    M, N, K = 8, 512, 4096
    x = torch.randn(M, K, device="cuda").to(t)
    Ws = [(torch.randn(N, K, device="cuda") * 0.05).to(t) for _ in range(4)]
    refs = [x.float() @ W.float().T for W in Ws]
    W = torch.zeros(N, K, device="cuda", dtype=t)
    Wt = torch.zeros(K, N, device="cuda", dtype=t)
    for n in range(40):
        W.copy_(Ws[n % 4])
        y = ops.linear_rows(W, x)
        Wt.copy_(Ws[n % 4].T)
        yt = ops.linear_rows(Wt.T, x, weights_settled=True)
        assert relerr(host(y), host(refs[n % 4])) <= BF16_TOL
        assert torch.equal(y, yt)


@pytest.mark.parametrize("B", [2, 3, 9, 16, 17])
def test_block_token_step_matches_separate_launches(ops, B):
    """The single-token launch sequences of a block against the same block cell by cell, on a carried state."""
    from xlstm_cuda.blocks import mLSTMBlock
    t = torch.bfloat16
    torch.manual_seed(B)
    with torch.device("cuda"):
        blk = mLSTMBlock(0, embedding_dim=512, num_heads=2, compute_dtype=t).to(t)
    blk.fuse_projections()
    x = torch.randn(B, 1, 512, device="cuda", dtype=t)
    st = (torch.randn(B, 2, 128, 256, device="cuda") * 0.1, torch.randn(B, 2, 128, device="cuda") * 0.1, torch.zeros(B, 2, device="cuda"))
    with torch.inference_mode():
        y, s1 = blk(x, st)
        out, s2 = blk.mlstm_cell(blk.norm_mlstm(x), st)
        x1, xn = ops.add_rms_norm(x, out, blk.norm_ffn.weight, blk.norm_ffn.eps)
        ref = x1 + blk.ffn_proj_down(ops.swiglu(blk.ffn_proj_up_gate(xn), blk.ffn_proj_up(xn)))
    assert relerr(host(y), host(ref)) <= BF16_TOL
    for a, b in zip(s1, s2):
        assert relerr(host(a), host(b)) <= BF16_TOL


@pytest.mark.parametrize("B", [4, 8])
def test_block_token_step_with_weights_at_odd_offsets(ops, B):
    """Weights that are views at an odd offset, or transposed: the streaming kernels do not take them, the block does."""
    m, _, _ = _blocks()
    x = torch.randn(B, 1, 512, device="cuda", dtype=torch.bfloat16)
    with torch.inference_mode():
        y = m(x)[0]
    out, down = m.mlstm_cell.output_cell.out_proj, m.ffn_proj_down
    down.weight.data = down.weight.data.T.contiguous().T
    if B > 4:
        flat = torch.empty(out.weight.numel() + 1, device="cuda", dtype=torch.bfloat16)
        flat[1:] = out.weight.data.reshape(-1)
        out.weight.data = flat[1:].view_as(out.weight)
    with torch.inference_mode():
        assert relerr(host(m(x)[0]), host(y)) <= BF16_TOL


@pytest.mark.parametrize("B", [3, 16])
@pytest.mark.parametrize("what", ["input", "norm_mlstm", "norm_ffn"])
def test_block_token_step_with_inputs_or_norms_at_odd_offsets(ops, B, what):
    """An input or a norm weight off a 16-byte boundary: the norm is a launch of its own, with the same bits."""
    m, _, _ = _blocks()
    x = torch.randn(B, 1, 512, device="cuda", dtype=torch.bfloat16)
    with torch.inference_mode():
        for mod in (m.norm_mlstm, m.norm_ffn):
            mod.weight.uniform_(0.5, 1.5)
        y, st = m(x)
        off = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)
        if what == "input":
            x = off(x)
        else:
            mod = getattr(m, what)
            mod.weight.data = off(mod.weight.data)
        y2, st2 = m(x)
        assert torch.equal(y, y2) and all(torch.equal(a, b) for a, b in zip(st, st2))


@pytest.mark.parametrize("d,NH,B", [(4096, 8, 5), (4096, 8, 16), (2048, 8, 16)])
def test_block_token_step_with_norms_of_their_own(ops, d, NH, B):
    """Rows beyond what the Linears take a norm for (48 KB): the norms are launches, in the same native call.  Against the block cell by
    cell, the state carried over several tokens."""
    from xlstm_cuda.blocks import mLSTMBlock
    t = torch.bfloat16
    assert B * (2 * d + 64) + 2 * d > 49152
    torch.manual_seed(B)
    with torch.device("cuda"):
        blk = mLSTMBlock(0, embedding_dim=d, num_heads=NH, compute_dtype=t).to(t)
    blk.fuse_projections()
    with torch.inference_mode():
        for mod in (blk.norm_mlstm, blk.norm_ffn):
            mod.weight.uniform_(0.5, 1.5)
        st = ref_st = None
        for _ in range(4):
            x = torch.randn(B, 1, d, device="cuda", dtype=t)
            y, st = blk(x, st)
            out, ref_st = blk.mlstm_cell(blk.norm_mlstm(x), ref_st)
            x1, xn = ops.add_rms_norm(x, out, blk.norm_ffn.weight, blk.norm_ffn.eps)
            ref = x1 + blk.ffn_proj_down(ops.swiglu(blk.ffn_proj_up_gate(xn), blk.ffn_proj_up(xn)))
            assert relerr(host(y), host(ref)) <= BF16_TOL
            for a, b in zip(st, ref_st):
                assert relerr(host(a), host(b)) <= BF16_TOL


def test_block_token_reports_the_call_that_failed(ops):
    """A weight that the Linear does not take (odd offset): the status comes with that Linear's name, for both kinds of it."""
    from xlstm_cuda._lib import XlstmCudaError
    m, _, _ = _blocks()
    cell = m.mlstm_cell
    W, b = cell._fused_weights()
    out, down, rk = cell.output_cell.out_proj, m.ffn_proj_down, cell.recurrent_kernel
    odd = torch.cat([out.weight.new_zeros(1), out.weight.detach().flatten()])[1:].view_as(out.weight)
    for B, rows, name in ((2, False, "xlstm_linear_token"), (8, True, "xlstm_linear_rows_norm")):
        with torch.inference_mode(), pytest.raises(XlstmCudaError, match=name):
            ops.mlstm_token_block(torch.zeros(B, 512, device="cuda", dtype=torch.bfloat16), W, b, (m.norm_mlstm.weight, 1e-6),
                                  (cell.num_heads, cell.qk_dim_per_head, cell.v_dim_per_head), None, (None, 1e-6), rk.eps, False, 15.0,
                                  (odd, None), (m.norm_ffn.weight, 1e-6), m._fused_ffn(), (down.weight, None), rows)


def _blocks():
    from xlstm_cuda.blocks import mLSTMBlock, sLSTMBlock, sLSTMBlockDiag
    t = torch.bfloat16
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = mLSTMBlock(0, embedding_dim=512, num_heads=2, compute_dtype=t).to(t)
        m.fuse_projections()
        s = sLSTMBlock(0, embedding_dim=512, num_heads=2).to(t)

        class Config:
            inp_dim, head_dim, head_num, p_factor, norm_eps, gate_soft_cap = 128, 64, 2, (2.0, 1.5), 1e-6, 15.0
        d = sLSTMBlockDiag(Config()).to(t)
    return m, s, d


@pytest.mark.parametrize("B", [8, 20])
def test_fused_launches_leave_hooks_and_replaced_modules_alone(ops, B):
    """Modules whose call a fused launch would leave out are called where somebody listens, or has put another module there."""
    m, s, _ = _blocks()
    x = torch.randn(B, 1, 512, device="cuda", dtype=torch.bfloat16)
    seen = []
    with torch.inference_mode():
        y, ys = m(x)[0], s(x)[0]
        for blk, mods in ((m, (m.norm_mlstm, m.mlstm_cell, m.mlstm_cell.recurrent_kernel, m.mlstm_cell.output_cell.out_proj,
                               m.ffn_proj_down)), (s, (s.norm_ffn,))):
            for mod in mods:
                handle = mod.register_forward_hook(lambda mod, args, out: seen.append(mod))
                out = blk(x)[0]
                handle.remove()
                assert seen == [mod] and relerr(host(out), host(y if blk is m else ys)) <= BF16_TOL
                seen.clear()

        class Doubled(torch.nn.Linear):
            def forward(self, x):
                return 2 * super().forward(x)
        with torch.device("cuda"):
            other = Doubled(512, 512, bias=False).to(torch.bfloat16)
        other.weight.copy_(m.mlstm_cell.output_cell.out_proj.weight * 0.5)
        m.mlstm_cell.output_cell.out_proj = other
        assert relerr(host(m(x)[0]), host(y)) <= BF16_TOL


def test_fused_launches_leave_gradients_alone(ops):
    """Where gradients are recorded the blocks reach the same parameters and inputs as their separate ops do."""
    m, s, d = _blocks()
    x = torch.randn(8, 1, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    s(x)[0].float().pow(2).sum().backward()
    assert x.grad is not None and s.slstm_cell.output_cell.out_proj.weight.grad is not None
    m(x)[0].float().pow(2).sum().backward()
    assert m.ffn_proj_down.weight.grad is not None
    xd = torch.randn(3, 5, 128, device="cuda", dtype=torch.bfloat16)
    y = d(xd)[0]
    y.float().pow(2).sum().backward()
    assert d.up_proj.weight.grad is not None and d.hid_norm.weight.grad is not None
    with torch.no_grad():
        assert relerr(host(d(xd)[0]), host(y)) <= BF16_TOL


def test_linear_token_rejects_what_it_does_not_do(ops):
    with pytest.raises(ValueError):
        ops.geglu(torch.zeros(4, 33, device="cuda"))
    t = torch.bfloat16
    with pytest.raises(ValueError):
        ops.linear_token(torch.zeros(8, 16, device="cuda", dtype=t), torch.zeros(5, 16, device="cuda", dtype=t))
    with pytest.raises(TypeError):
        ops.linear_token(torch.zeros(8, 16, device="cuda"), torch.zeros(1, 16, device="cuda"))
    with pytest.raises(ValueError):
        ops.linear_rows(torch.zeros(8, 32, device="cuda", dtype=t), torch.zeros(17, 32, device="cuda", dtype=t))
