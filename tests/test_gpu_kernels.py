"""GPU parity: every kernel through the C ABI against the CPU oracle and the golden fixtures.

Tolerances (max|a-b| / max|b|): fp32 1e-4 on h, C, n and 1e-4 absolute on m;
bf16 activations with fp32 state 2e-2.
"""
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

from conftest import relerr
from oracle import oracle as xo

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-4
BF16_TOL = 2e-2


def dev(a, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def host(t):
    return t.detach().float().cpu().numpy()


def gates(rng, shape, fmean=3.0):
    i = 15.0 * np.tanh(rng.standard_normal(shape).astype(np.float32) / 15.0)
    f = 15.0 * np.tanh((rng.standard_normal(shape).astype(np.float32) + fmean) / 15.0)
    return i, f


@pytest.fixture(scope="module")
def ops():
    from xlstm_cuda import ops as _ops
    return _ops


# ---- soft-cap ----------------------------------------------------------------
@pytest.mark.parametrize("n", [1, 7, 4096, 50304, 1 << 20 | 3])
@pytest.mark.parametrize("cap", [15.0, 30.0])
def test_softcap_fp32(ops, n, cap):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 20).astype(np.float32)
    y = host(ops.softcap(dev(x), cap))
    np.testing.assert_allclose(y, xo.softcap(x, cap), rtol=1e-5, atol=1e-5)


def test_softcap_bf16_and_unaligned_and_kat(ops, golden):
    rng = np.random.default_rng(0)
    x = xo.bf16_round((rng.standard_normal(10001) * 20).astype(np.float32))
    y = host(ops.softcap(dev(x, torch.bfloat16), 30.0))
    assert relerr(y, xo.softcap(x, 30.0)) < 4e-3
    base = dev(np.arange(1003, dtype=np.float32) / 10 - 50)
    view = base[1:]  # 4-byte aligned only
    np.testing.assert_allclose(host(ops.softcap(view, 15.0)), xo.softcap(host(view), 15.0), rtol=1e-5, atol=1e-5)
    g = golden("kat")
    for tag in ("small", "large", "edge"):
        y = host(ops.softcap(dev(g[f"softcap_{tag}_x"]), float(g[f"softcap_{tag}_cap"])))
        np.testing.assert_allclose(y, g[f"softcap_{tag}_y"], rtol=1e-6, atol=1e-6)
    x = dev(np.ones(5, np.float32))
    assert ops.softcap(x, None) is x and ops.softcap(x, 0.0) is x
    assert ops.softcap(torch.empty(0, device="cuda"), 15.0).numel() == 0


# ---- decode step ------------------------------------------------------------------
def run_steps(ops, g, dtype, inplace=False):
    st = (dev(g["C0"]), dev(g["n0"]), dev(g["m0"]))
    hs = []
    for t in range(g["q"].shape[2]):
        a = [dev(g[x][:, :, t], dtype) for x in "qkvif"]
        h, st = ops.mlstm_step(*a, state=st, inplace=inplace)
        hs.append(host(h))
    return np.stack(hs, 2), tuple(host(s) for s in st)


@pytest.mark.parametrize("name", ["mlstm_step_bf16", "mlstm_step_7b"])
def test_mlstm_step_against_reference_fixture(ops, golden, name):
    g = golden(name)
    # fp32 activations (bf16-representable values): 1e-4 against the reference's fp32 run
    h, (C, n, m) = run_steps(ops, g, torch.float32)
    assert relerr(h, g["h_fp32"]) < FP32_TOL and relerr(C, g["C_fp32"]) < FP32_TOL
    assert relerr(n, g["n_fp32"]) < FP32_TOL and np.abs(m - g["m_fp32"]).max() < FP32_TOL
    # bf16 activations, fp32 state: 2e-2 against the reference's bf16-compute run and its fp32 run
    h, (C, n, m) = run_steps(ops, g, torch.bfloat16, inplace=True)
    assert relerr(h, g["h_bf16"]) < BF16_TOL and relerr(h, g["h_fp32"]) < BF16_TOL
    assert relerr(C, g["C_bf16"]) < BF16_TOL and relerr(n, g["n_bf16"]) < BF16_TOL
    assert np.abs(m - g["m_bf16"]).max() < BF16_TOL


@pytest.mark.parametrize("B,NH,dqk,dv", [(16, 8, 256, 512), (3, 5, 64, 64), (2, 2, 100, 36), (1, 1, 512, 1024)])
def test_mlstm_step_against_oracle(ops, B, NH, dqk, dv):
    rng = np.random.default_rng(B * 1000 + dqk)
    q, k = (rng.standard_normal((B, NH, 1, dqk)).astype(np.float32) for _ in range(2))
    v = rng.standard_normal((B, NH, 1, dv)).astype(np.float32)
    i, f = gates(rng, (B, NH, 1))
    st = (rng.standard_normal((B, NH, dqk, dv)).astype(np.float32) * 0.1,
          rng.standard_normal((B, NH, dqk)).astype(np.float32) * 0.1, rng.standard_normal((B, NH)).astype(np.float32))
    for state in (st, None):
        h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f, state)
        h, st_new = ops.mlstm_step(dev(q[:, :, 0]), dev(k[:, :, 0]), dev(v[:, :, 0]), dev(i[:, :, 0]), dev(f[:, :, 0]),
                                   None if state is None else tuple(dev(s) for s in state))
        assert relerr(host(h), h_ref[:, :, 0]) < FP32_TOL
        for got, want in zip(st_new, st_ref):
            assert relerr(host(got), want) < FP32_TOL


def test_mlstm_step_config2_256_steps_bf16(ops):
    """Decode of a serving batch: B=16, NH=8, 256/512, bf16 activations, fp32 state, 256 carried steps."""
    B, NH, dqk, dv, T = 16, 8, 256, 512, 256
    g = torch.Generator().manual_seed(1)
    C = torch.randn(B, NH, dqk, dv, generator=g) * 0.1
    n = torch.randn(B, NH, dqk, generator=g) * 0.1
    m = torch.zeros(B, NH)
    q = torch.randn(B, NH, T, dqk, generator=g).bfloat16()
    k = torch.randn(B, NH, T, dqk, generator=g).bfloat16()
    v = torch.randn(B, NH, T, dv, generator=g).bfloat16()
    i = (15 * torch.tanh(torch.randn(B, NH, T, generator=g) / 15)).bfloat16()
    f = (15 * torch.tanh((torch.randn(B, NH, T, generator=g) + 3) / 15)).bfloat16()
    h_ref, st_ref = xo.mlstm_recurrent(q.float().numpy(), k.float().numpy(), v.float().numpy(), i.float().numpy(),
                                       f.float().numpy(), (C.numpy(), n.numpy(), m.numpy()))
    st = (C.cuda(), n.cuda(), m.cuda())
    qd, kd, vd, idv, fd = (t.cuda() for t in (q, k, v, i, f))
    hs = []
    for t in range(T):
        h, st = ops.mlstm_step(qd[:, :, t], kd[:, :, t], vd[:, :, t], idv[:, :, t], fd[:, :, t], st, inplace=True)
        hs.append(h)
    h = host(torch.stack(hs, 2))
    assert relerr(h, h_ref) < BF16_TOL
    assert relerr(host(st[0]), st_ref[0]) < FP32_TOL * 10 and relerr(host(st[1]), st_ref[1]) < FP32_TOL * 10
    assert np.abs(host(st[2]) - st_ref[2]).max() < 1e-3


def test_mlstm_step_layer_ring_overlapped_launches(ops):
    """A stack of layers stepped token by token with state_settled=True (each launch may start fetching its
    state while the launch before it - another layer - drains), eagerly and replayed as a CUDA graph, against
    the oracle stepping every layer on its own; and the same state stepped twice in a row WITHOUT the promise."""
    B, NH, dqk, dv, LAYERS, T = 2, 4, 128, 256, 3, 6
    rng = np.random.default_rng(77)
    q, k = (rng.standard_normal((LAYERS, B, NH, T, dqk)).astype(np.float32) for _ in range(2))
    v = rng.standard_normal((LAYERS, B, NH, T, dv)).astype(np.float32)
    i, f = gates(rng, (LAYERS, B, NH, T))
    st0 = [(rng.standard_normal((B, NH, dqk, dv)).astype(np.float32) * 0.1,
            rng.standard_normal((B, NH, dqk)).astype(np.float32) * 0.1, np.zeros((B, NH), np.float32)) for _ in range(LAYERS)]
    ref = [xo.mlstm_recurrent(q[l], k[l], v[l], i[l], f[l], st0[l]) for l in range(LAYERS)]
    qd, kd, vd, idv, fd = (dev(a) for a in (q, k, v, i, f))

    def run(states, hs):
        for t in range(T):
            for l in range(LAYERS):
                h, states[l] = ops.mlstm_step(qd[l, :, :, t], kd[l, :, :, t], vd[l, :, :, t], idv[l, :, :, t], fd[l, :, :, t],
                                              states[l], state_settled=True)
                hs[l][:, :, t] = h

    states = [tuple(dev(a) for a in st) for st in st0]
    hs = [torch.empty(B, NH, T, dv, device="cuda") for _ in range(LAYERS)]
    run(states, hs)
    for l in range(LAYERS):
        assert relerr(host(hs[l]), ref[l][0]) < FP32_TOL
        for got, want in zip(states[l], ref[l][1]):
            assert relerr(host(got), want) < FP32_TOL

    # the same launches as one CUDA graph (the decode loop's form): bit-identical to the eager run
    states_g = [tuple(dev(a) for a in st) for st in st0]
    hs_g = [torch.empty(B, NH, T, dv, device="cuda") for _ in range(LAYERS)]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    final = []
    with torch.cuda.graph(graph, stream=side):
        work = list(states_g)
        run(work, hs_g)
        final = work
    torch.cuda.current_stream().wait_stream(side)
    graph.replay()
    torch.cuda.synchronize()
    for l in range(LAYERS):
        assert torch.equal(hs_g[l], hs[l])
        for got, want in zip(final[l], states[l]):
            assert torch.equal(got, want)

    # one state stepped T times back to back, no promise: every launch reads what the one before it wrote
    st = tuple(dev(a) for a in st0[0])
    out = []
    for t in range(T):
        h, st = ops.mlstm_step(qd[0, :, :, t], kd[0, :, :, t], vd[0, :, :, t], idv[0, :, :, t], fd[0, :, :, t], st, inplace=True)
        out.append(h)
    assert relerr(host(torch.stack(out, 2)), ref[0][0]) < FP32_TOL


@pytest.mark.parametrize("group", [1, 3])
def test_decode_pipeline_host_fed(ops, group):
    """runtime.DecodePipeline: pinned host q,k,v,i,f in, h out, every step; eager enqueue and the captured graph
    (steps travelling in groups) must both reproduce the plain decode step bit for bit, states included."""
    from xlstm_cuda.runtime import DecodePipeline
    B, NH, dqk, dv, LAYERS, T = 2, 4, 128, 256, 3, 4
    g = torch.Generator().manual_seed(5)
    steps = LAYERS * T
    q = torch.randn(steps, B, NH, dqk, generator=g).bfloat16()
    k = torch.randn(steps, B, NH, dqk, generator=g).bfloat16()
    v = torch.randn(steps, B, NH, dv, generator=g).bfloat16()
    i = torch.randn(steps, B, NH, generator=g).bfloat16()
    f = (torch.randn(steps, B, NH, generator=g) + 3).bfloat16()

    def fresh_states():
        gs = torch.Generator().manual_seed(6)
        return [[(torch.randn(B, NH, dqk, dv, generator=gs).cuda() * 0.1, torch.randn(B, NH, dqk, generator=gs).cuda() * 0.1,
                  torch.zeros(B, NH, device="cuda")),
                 tuple(torch.empty(s, device="cuda") for s in ((B, NH, dqk, dv), (B, NH, dqk), (B, NH)))] for _ in range(LAYERS)]

    # reference: the plain op, layer by layer
    st = [s[0] for s in fresh_states()]
    h_ref = []
    for t in range(steps):
        l = t % LAYERS
        h, st[l] = ops.mlstm_step(q[t].cuda(), k[t].cuda(), v[t].cuda(), i[t].cuda(), f[t].cuda(), st[l])
        h_ref.append(h)

    for captured in (False, True):
        pipe = DecodePipeline(B, NH, dqk, dv, "cuda", group=group)
        packed = [pipe.pack(q[t], k[t], v[t], i[t], f[t]) for t in range(steps)]
        h_host = [torch.empty(B, NH, dv, dtype=torch.bfloat16).pin_memory() for _ in range(steps)]
        states = fresh_states()
        side = [0] * LAYERS
        items = []
        for t in range(steps):
            l = t % LAYERS
            items.append((packed[t], states[l][side[l]], states[l][side[l] ^ 1], h_host[t], True))
            side[l] ^= 1
        if captured:
            graph = pipe.capture(items)
            graph.replay()
            torch.cuda.synchronize()
        else:
            for lo in range(0, steps, group):
                pipe.step_group(items[lo:lo + group])
            pipe.synchronize()
        for t in range(steps):
            assert torch.equal(h_host[t], h_ref[t].cpu()), (captured, t)
        for l in range(LAYERS):
            for got, want in zip(states[l][side[l]], st[l]):
                assert torch.equal(got, want)


@pytest.mark.parametrize("B,NH,dqk,dv", [(2, 4, 128, 256), (1, 8, 256, 512), (3, 2, 64, 96)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mlstm_step_with_fused_output_epilogue(ops, B, NH, dqk, dv, dtype):
    """xlstm_mlstm_step_gated (norm x weight x sigmoid(output gate) applied inside the step kernel, the head's
    CTAs meeting through their cluster) against the two separate kernels and against the oracle; the output gate
    is handed over as a column block of a wider projection output, as the block does."""
    rng = np.random.default_rng(B * 100 + dv)
    rnd = (lambda a: xo.bf16_round(a)) if dtype == torch.bfloat16 else (lambda a: a)
    q, k = (rnd(rng.standard_normal((B, NH, dqk)).astype(np.float32)) for _ in range(2))
    v = rnd(rng.standard_normal((B, NH, dv)).astype(np.float32))
    i, f = (rnd(a[:, :, 0]) for a in gates(rng, (B, NH, 1)))
    wide = rnd(rng.standard_normal((B, NH * dv + 24)).astype(np.float32) * 2.0)
    og = wide[:, 16:16 + NH * dv]
    w = rnd(rng.uniform(0.5, 1.5, NH * dv).astype(np.float32))
    st = (rng.standard_normal((B, NH, dqk, dv)).astype(np.float32) * 0.1,
          rng.standard_normal((B, NH, dqk)).astype(np.float32) * 0.1, rng.standard_normal((B, NH)).astype(np.float32))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dtype).cuda()
    wide_d = d(wide)
    for state in (st, None):
        sd = None if state is None else tuple(dev(x) for x in state)
        h, st_ref = ops.mlstm_step(d(q), d(k), d(v), d(i), d(f), sd)
        y_ref = ops.mlstm_output_gate(h.unsqueeze(2), wide_d[:, 16:16 + NH * dv].unsqueeze(1), d(w), 1e-6)[:, 0]
        y, st_new = ops.mlstm_step_gated(d(q), d(k), d(v), d(i), d(f), wide_d[:, 16:16 + NH * dv], d(w), sd, norm_eps=1e-6)
        tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
        assert y.shape == (B, NH * dv) and relerr(host(y), host(y_ref)) <= tol
        for got, want in zip(st_new, st_ref):
            assert torch.equal(got, want)
        # and against the oracle: recurrent step, then the epilogue restated on the host
        h_o, _ = xo.mlstm_recurrent(q[:, :, None], k[:, :, None], v[:, :, None], i[:, :, None], f[:, :, None], state)
        y_o = xo.mlstm_output_gate(rnd(h_o), og[:, None, :], w, 1e-6)[:, 0]
        assert relerr(host(y), y_o) <= tol * (1 if dtype == torch.float32 else 2)


# ---- chunkwise -------------------------------------------------------------------
def test_chunkwise_config1_fp32(ops, golden):
    g = golden("mlstm_c1_fp32")
    for L in (64, 32, 128):   # 128: beyond the exact kernel's tile, walked in tiles of 64
        h, st = ops.mlstm_chunkwise(*(dev(g[x]) for x in "qkvif"), state=None, chunk_size=L)
        assert relerr(host(h), g["h"]) < FP32_TOL
        assert relerr(host(st[0]), g["C"]) < FP32_TOL and relerr(host(st[1]), g["n"]) < FP32_TOL
        assert np.abs(host(st[2]) - g["m"]).max() < FP32_TOL


def test_chunkwise_ragged_with_state_fp32(ops, golden):
    g = golden("mlstm_ragged_fp32")
    st0 = tuple(dev(g[x]) for x in ("C0", "n0", "m0"))
    for L in (64, 16, 7):
        h, st = ops.mlstm_chunkwise(*(dev(g[x]) for x in "qkvif"), state=st0, chunk_size=L)
        assert relerr(host(h), g["h"]) < FP32_TOL
        assert relerr(host(st[0]), g["C"]) < FP32_TOL and relerr(host(st[1]), g["n"]) < FP32_TOL
        assert np.abs(host(st[2]) - g["m"]).max() < FP32_TOL


@pytest.mark.parametrize("B,NH,S,dqk,dv", [(1, 2, 128, 256, 512), (2, 1, 70, 128, 192), (1, 1, 1, 64, 64)])
def test_chunkwise_against_oracle_and_strided_inputs(ops, B, NH, S, dqk, dv):
    rng = np.random.default_rng(S)
    # projection-style layout [B,S,NH,d], handed over as a permuted view
    q, k = (rng.standard_normal((B, S, NH, dqk)).astype(np.float32) for _ in range(2))
    v = rng.standard_normal((B, S, NH, dv)).astype(np.float32)
    i, f = gates(rng, (B, S, NH))
    tr = lambda a: np.ascontiguousarray(np.moveaxis(a, 1, 2))
    h_ref, st_ref = xo.mlstm_recurrent(tr(q), tr(k), tr(v), tr(i), tr(f))
    h, st = ops.mlstm_chunkwise(dev(q).permute(0, 2, 1, 3), dev(k).permute(0, 2, 1, 3), dev(v).permute(0, 2, 1, 3),
                                dev(i).permute(0, 2, 1), dev(f).permute(0, 2, 1))
    assert relerr(host(h), h_ref) < FP32_TOL
    for got, want in zip(st, st_ref):
        assert relerr(host(got), want) < FP32_TOL
    # run twice: bitwise identical
    h2, _ = ops.mlstm_chunkwise(dev(q).permute(0, 2, 1, 3), dev(k).permute(0, 2, 1, 3), dev(v).permute(0, 2, 1, 3),
                                dev(i).permute(0, 2, 1), dev(f).permute(0, 2, 1))
    assert torch.equal(h, h2)


def test_chunkwise_equals_steps_and_split_sequence(ops):
    """chunkwise(S) == S decode steps == chunkwise(S1) then chunkwise(S2) with the carried state."""
    rng = np.random.default_rng(5)
    B, NH, S, dqk, dv = 2, 2, 96, 64, 128
    q, k = (dev(rng.standard_normal((B, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = dev(rng.standard_normal((B, NH, S, dv)).astype(np.float32))
    i, f = (dev(a) for a in gates(rng, (B, NH, S)))
    h, st = ops.mlstm_chunkwise(q, k, v, i, f)
    h1, st1 = ops.mlstm_chunkwise(q[:, :, :50], k[:, :, :50], v[:, :, :50], i[:, :, :50], f[:, :, :50])
    h2, st2 = ops.mlstm_chunkwise(q[:, :, 50:], k[:, :, 50:], v[:, :, 50:], i[:, :, 50:], f[:, :, 50:], st1)
    assert relerr(host(torch.cat([h1, h2], 2)), host(h)) < FP32_TOL
    assert relerr(host(st2[0]), host(st[0])) < FP32_TOL
    s, hs = None, []
    for t in range(S):
        ht, s = ops.mlstm_step(q[:, :, t], k[:, :, t], v[:, :, t], i[:, :, t], f[:, :, t], s)
        hs.append(ht)
    assert relerr(host(torch.stack(hs, 2)), host(h)) < FP32_TOL
    assert relerr(host(s[0]), host(st[0])) < FP32_TOL and np.abs(host(s[2]) - host(st[2])).max() < FP32_TOL


def test_chunkwise_bf16_head_shape(ops):
    rng = np.random.default_rng(8)
    B, NH, S, dqk, dv = 1, 2, 256, 256, 512
    q, k = (xo.bf16_round(rng.standard_normal((B, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = xo.bf16_round(rng.standard_normal((B, NH, S, dv)).astype(np.float32))
    i, f = (xo.bf16_round(a) for a in gates(rng, (B, NH, S)))
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f)
    h, st = ops.mlstm_chunkwise(*(dev(a, torch.bfloat16) for a in (q, k, v, i, f)))
    assert relerr(host(h), h_ref) < BF16_TOL
    assert relerr(host(st[0]), st_ref[0]) < BF16_TOL and relerr(host(st[1]), st_ref[1]) < BF16_TOL
    assert np.abs(host(st[2]) - st_ref[2]).max() < BF16_TOL


def recurrent_fp64(q, k, v, i, f, eps=1e-6):
    """The recurrence in float64 (numpy), for inputs where fp32 itself is the limit."""
    q, k, v, i, f = (a.astype(np.float64) for a in (q, k, v, i, f))
    B, NH, S, dqk = q.shape
    C = np.zeros((B, NH, dqk, v.shape[-1])); n = np.zeros((B, NH, dqk)); m = np.zeros((B, NH)); hs = []
    for t in range(S):
        fl = -np.logaddexp(0, -f[:, :, t])
        mn = np.maximum(fl + m, i[:, :, t])
        fg, ig = np.exp(fl + m - mn), np.exp(i[:, :, t] - mn)
        C = fg[..., None, None] * C + ig[..., None, None] * k[:, :, t, :, None] * v[:, :, t, None, :]
        n = fg[..., None] * n + ig[..., None] * k[:, :, t]
        m = mn
        qs = q[:, :, t] / np.sqrt(dqk)
        den = np.maximum(np.abs(np.einsum("bhd,bhd->bh", qs, n)), np.exp(-m)) + eps
        hs.append(np.einsum("bhd,bhdv->bhv", qs, C) / den[..., None])
    return np.stack(hs, 2), (C, n, m)


def test_extreme_gates_stay_finite(ops):
    """Gates at the soft-cap limits (+-15) over many chunks: no inf/nan.  Here the fp32 recurrence
    itself is 1.2e-4 away from exact arithmetic (sums near 1e3 inside exp), so the kernel is held to
    1e-4 against a float64 evaluation and to 5e-4 against the fp32 oracle."""
    rng = np.random.default_rng(3)
    B, NH, S, dqk, dv = 1, 2, 192, 64, 64
    q, k = (rng.standard_normal((B, NH, S, dqk)).astype(np.float32) for _ in range(2))
    v = rng.standard_normal((B, NH, S, dv)).astype(np.float32)
    i = rng.choice([-15.0, 0.0, 15.0], size=(B, NH, S)).astype(np.float32)
    f = rng.choice([-15.0, 0.0, 15.0], size=(B, NH, S)).astype(np.float32)
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f)
    h64, st64 = recurrent_fp64(q, k, v, i, f)
    h, st = ops.mlstm_chunkwise(*(dev(a) for a in (q, k, v, i, f)))
    assert np.isfinite(host(h)).all()
    assert relerr(host(h), h64) < FP32_TOL and relerr(host(st[0]), st64[0]) < FP32_TOL
    assert relerr(host(h), h_ref) < 5e-4 and relerr(host(st[0]), st_ref[0]) < 5e-4
    assert np.abs(host(st[2]) - st_ref[2]).max() < 1e-3


def test_chunkwise_bf16_extreme_gates_tensor_core_path(ops):
    """bf16 tensor-core path with gates pinned at the soft-cap limits for long stretches: every exponent is a
    non-positive difference and the TMEM state is rescaled lazily, so nothing may overflow.  The final state
    must meet the bf16 tolerance against the float64 recurrence.  With such gates the normaliser q.n + sum(P)
    of many tokens is a near-cancellation (|h| reaches 1e4): there h = num/den amplifies the bf16 rounding of
    the weights by 1/|den| in ANY bf16 implementation, so h is compared on the well-conditioned tokens
    (|h| <= 5 in the float64 result, the usual range of h; 62 % of the tokens here) and only checked for finiteness elsewhere."""
    rng = np.random.default_rng(13)
    B, NH, S, dqk, dv = 1, 2, 768, 256, 256
    q, k = (xo.bf16_round(rng.standard_normal((B, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = xo.bf16_round(rng.standard_normal((B, NH, S, dv)).astype(np.float32))
    i = np.repeat(rng.choice([-15.0, 0.0, 15.0], size=(B, NH, S // 16)), 16, axis=-1).astype(np.float32)
    f = np.repeat(rng.choice([-15.0, 3.0, 15.0], size=(B, NH, S // 32), p=[0.1, 0.5, 0.4]), 32, axis=-1).astype(np.float32)
    h64, st64 = recurrent_fp64(q, k, v, i, f)
    bf = torch.bfloat16
    assert ops.chunkwise_workspace_bytes(B, NH, S, dqk, dv, 64, bf) > 0  # really the tensor-core path
    h, st = ops.mlstm_chunkwise(*(dev(a, bf) for a in (q, k, v, i, f)))
    assert np.isfinite(host(h)).all() and np.isfinite(host(st[0])).all()
    ok = np.abs(h64).max(axis=-1, keepdims=True) <= 5.0
    assert ok.mean() > 0.5
    assert relerr(np.where(ok, host(h), 0.0), np.where(ok, h64, 0.0)) < BF16_TOL
    assert relerr(host(st[0]), st64[0]) < BF16_TOL and relerr(host(st[1]), st64[1]) < BF16_TOL
    assert np.abs(host(st[2]) - st64[2]).max() < 1e-3


def test_chunkwise_full_length_properties(ops):
    """Full length (S = 32768, 256/512, bf16): the oracle cannot run this in seconds, so check
    (a) the first 384 tokens against the oracle, (b) one pass == two half passes with the carried state,
    (c) run-to-run bitwise determinism."""
    B, NH, S, dqk, dv = 1, 4, 32768, 256, 512
    g = torch.Generator().manual_seed(3)
    bf = torch.bfloat16
    q = torch.randn(B, NH, S, dqk, generator=g).to(bf)
    k = torch.randn(B, NH, S, dqk, generator=g).to(bf)
    v = torch.randn(B, NH, S, dv, generator=g).to(bf)
    i = (15 * torch.tanh(torch.randn(B, NH, S, generator=g) / 15)).to(bf)
    f = (15 * torch.tanh((torch.randn(B, NH, S, generator=g) + 3) / 15)).to(bf)
    P = 384
    h_ref, _ = xo.mlstm_recurrent(*(t[:, :, :P].float().numpy() for t in (q, k, v, i, f)))
    qd, kd, vd, idv, fd = (t.cuda() for t in (q, k, v, i, f))
    h, st = ops.mlstm_chunkwise(qd, kd, vd, idv, fd)
    assert relerr(host(h[:, :, :P]), h_ref) < BF16_TOL
    H = S // 2
    h1, st1 = ops.mlstm_chunkwise(qd[:, :, :H], kd[:, :, :H], vd[:, :, :H], idv[:, :, :H], fd[:, :, :H])
    h2, st2 = ops.mlstm_chunkwise(qd[:, :, H:], kd[:, :, H:], vd[:, :, H:], idv[:, :, H:], fd[:, :, H:], st1)
    assert relerr(host(torch.cat([h1, h2], 2)), host(h)) < BF16_TOL
    assert relerr(host(st2[0]), host(st[0])) < BF16_TOL and np.abs(host(st2[2]) - host(st[2])).max() < 1e-3
    assert torch.isfinite(h.float()).all()
    h_again, _ = ops.mlstm_chunkwise(qd, kd, vd, idv, fd)
    assert torch.equal(h, h_again)


@pytest.mark.parametrize("B,NH,S,dqk,dv,dtype,with_state", [
    (1, 2, 65, 20, 36, torch.float32, True),       # partial pieces of dqk and dv, one token in the second chunk
    (1, 4, 64, 64, 64, torch.float32, False),      # one chunk: no scratch
    (2, 3, 31, 128, 256, torch.float32, True),     # less than one state tile
    (1, 2, 200, 256, 192, torch.float32, False),   # 64-column CTAs, ragged last chunk
    (2, 8, 1606, 256, 512, torch.float32, True),   # 128-column CTAs, a second group of chunks continuing in place
    (1, 2, 130, 64, 128, torch.bfloat16, True),    # bf16 head shape outside the tensor-core kernels
    (1, 2, 130, 640, 128, torch.float32, True),    # heads beyond the 512 rows of the one-kernel form
])
def test_chunkwise_fp32_two_kernels(ops, B, NH, S, dqk, dv, dtype, with_state):
    """The fp32 forward at the edges of its tiles, chunks and groups, against the step-by-step oracle."""
    rng = np.random.default_rng(S + dqk)
    rnd = xo.bf16_round if dtype == torch.bfloat16 else (lambda a: a)
    q, k = (rnd(rng.standard_normal((B, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = rnd(rng.standard_normal((B, NH, S, dv)).astype(np.float32))
    i, f = (rnd(a) for a in gates(rng, (B, NH, S)))
    st0 = None
    if with_state:
        st0 = ((rng.standard_normal((B, NH, dqk, dv)) * 0.1).astype(np.float32),
               (rng.standard_normal((B, NH, dqk)) * 0.1).astype(np.float32), rng.standard_normal((B, NH)).astype(np.float32))
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f, st0)
    st = None if st0 is None else tuple(dev(a) for a in st0)
    h, st1 = ops.mlstm_chunkwise(*(dev(a, dtype) for a in (q, k, v, i, f)), state=st)
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    assert relerr(host(h), h_ref) < tol
    for a, r in zip(st1, st_ref):
        assert relerr(host(a), r) < FP32_TOL


@pytest.mark.parametrize("NH,S,dqk,dv", [(48, 50, 128, 256), (32, 65, 128, 256), (40, 130, 128, 256), (16, 600, 128, 256), (60, 130, 72, 200)])
def test_chunkwise_fp32_heads_do_not_depend_on_how_many_there_are(ops, NH, S, dqk, dv):
    """The number of heads decides on the columns of a CTA, of the states and of the outputs (128 and 128 in one chunk; 128 and 64;
    128 and 128; 64 and 128; the last part of dv in half a CTA), and on when the output kernel starts: bit for bit a head of its own."""
    torch.manual_seed(S)
    q, k, v = (torch.randn(1, NH, S, d, device="cuda") for d in (dqk, dqk, dv))
    i, f = torch.randn(1, NH, S, device="cuda"), torch.randn(1, NH, S, device="cuda") + 3
    st = (torch.randn(1, NH, dqk, dv, device="cuda"), torch.randn(1, NH, dqk, device="cuda"), torch.randn(1, NH, device="cuda"))
    for _ in range(3):
        h, s1 = ops.mlstm_chunkwise(q, k, v, i, f, st)
        for n in (0, NH // 2, NH - 1):
            one = slice(n, n + 1)
            ho, so = ops.mlstm_chunkwise(*(a[:, one] for a in (q, k, v, i, f)), tuple(s[:, one].contiguous() for s in st))
            assert torch.equal(h[:, one], ho) and all(torch.equal(a[:, one], b) for a, b in zip(s1, so))


def test_chunkwise_fp32_normaliser_of_one_token_is_rounded_once(ops):
    """With an input gate that weighs the token with exactly one, n' = decay n + k is one multiply-add: bit for bit the float64
    value rounded to fp32, for the decay that the kernel itself uses (read off n = 1, k = 0)."""
    torch.manual_seed(0)
    NH, dqk, dv = 3, 256, 64
    k, n, v = torch.randn(1, NH, 1, dqk, device="cuda"), torch.randn(1, NH, dqk, device="cuda"), torch.randn(1, NH, 1, dv, device="cuda")
    i, f, m, C = (torch.zeros(1, NH, 1, device="cuda"), torch.randn(1, NH, 1, device="cuda"), torch.zeros(1, NH, device="cuda"),
                  torch.zeros(1, NH, dqk, dv, device="cuda"))
    after = lambda k, n: ops.mlstm_chunkwise(k, k, v, i, f, (C, n, m))[1][1]
    decay = after(torch.zeros_like(k), torch.ones_like(n))
    assert bool((decay < 1).all())
    assert torch.equal(after(k, n), (decay.double() * n.double() + k[:, :, 0].double()).float())


# ---- sLSTM ------------------------------------------------------------------------
@pytest.mark.parametrize("tag", ["a", "b", "x", "z"])
def test_slstm_scan_fixture(ops, golden, tag):
    g = golden("slstm_a")
    st = None if tag == "z" else tuple(dev(g[f"{tag}_{s}0"]) for s in "cnm")
    h, (c, n, m) = ops.slstm_scan(*(dev(g[f"{tag}_{x}"]) for x in "zifo"), state=st)
    tol = 1e-4 if tag == "x" else 1e-5
    assert relerr(host(h), g[f"{tag}_h"]) < tol and relerr(host(c), g[f"{tag}_c"]) < tol
    assert relerr(host(n), g[f"{tag}_n"]) < tol and np.abs(host(m) - g[f"{tag}_m"]).max() < tol


@pytest.mark.parametrize("B,S,NH,H,dtype", [(32, 100, 4, 256, torch.float32), (3, 33, 2, 40, torch.float32),
                                             (2, 64, 4, 1024, torch.float32), (4, 70, 4, 256, torch.bfloat16)])
def test_slstm_scan_oracle(ops, B, S, NH, H, dtype):
    rng = np.random.default_rng(H + S)
    rd = xo.bf16_round if dtype == torch.bfloat16 else (lambda a: a)
    z = rd(rng.standard_normal((B, S, NH, H)).astype(np.float32))
    i, f = (rd(a) for a in gates(rng, (B, S, NH)))
    o = rd(rng.standard_normal((B, S, NH)).astype(np.float32))
    h_ref, st_ref = xo.slstm_scan(z, i, f, o)
    h, st = ops.slstm_scan(*(dev(a, dtype) for a in (z, i, f, o)))
    tol = BF16_TOL if dtype == torch.bfloat16 else FP32_TOL
    assert relerr(host(h), h_ref) < tol
    for got, want in zip(st, st_ref):
        assert relerr(host(got), want) < FP32_TOL


@pytest.mark.parametrize("B,S,NH,H,dtype,with_state", [
    (1, 95, 1, 64, torch.float32, False),     # two gate tiles: one pass
    (1, 97, 2, 128, torch.float32, True),     # three segments, the last one a single step
    (1, 1000, 2, 1024, torch.float32, True),  # many segments, several unit slices, ragged end
    (2, 333, 1, 37, torch.float32, False),    # width without 16-byte vectors
    (1, 1024, 4, 40, torch.bfloat16, True),   # a slice with idle lanes
    (1, 200, 2, 1028, torch.float32, True),   # more than 1024 units
])
def test_slstm_scan_segments(ops, B, S, NH, H, dtype, with_state):
    """Segments of the sequence in parallel against the oracle, raw gates capped inside, and an in-place state (which
    takes the single pass) through the C ABI."""
    rng = np.random.default_rng(S)
    rnd = (lambda a: xo.bf16_round(a)) if dtype == torch.bfloat16 else (lambda a: a)
    z = rnd(rng.standard_normal((B, S, NH, H)).astype(np.float32))
    i, f, o = (rnd((rng.standard_normal((B, S, NH)) * 3 + s).astype(np.float32)) for s in (0, 2, 0))
    st0 = None
    if with_state:
        st0 = (rng.standard_normal((B, NH, H)).astype(np.float32), rng.uniform(0.5, 2, (B, NH, H)).astype(np.float32),
               rng.standard_normal((B, NH)).astype(np.float32))
    cap = 5.0
    h_ref, st_ref = xo.slstm_scan(z, *(xo.softcap(g, cap) for g in (i, f, o)), st0)
    st = None if st0 is None else tuple(dev(s) for s in st0)
    args = [dev(a, dtype) for a in (z, i, f, o)]
    h, st1 = ops.slstm_scan(*args, state=st, gate_cap=cap)
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    assert relerr(host(h), h_ref) < tol
    for a, r in zip(st1, st_ref):
        assert relerr(host(a), r) < tol
    if st is not None:
        from xlstm_cuda import _lib
        c, n, m1 = st[0].clone(), st[1].clone(), torch.empty_like(st[2])
        h2 = torch.empty_like(h)
        code = _lib.F32 if dtype == torch.float32 else _lib.BF16
        need = _lib.load().xlstm_slstm_scan_workspace_bytes(B, S, NH, H, code)
        assert need > 0
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        rc = _lib.load().xlstm_slstm_scan_ex(*(a.data_ptr() for a in args), c.data_ptr(), n.data_ptr(), st[2].data_ptr(),
                                             h2.data_ptr(), c.data_ptr(), n.data_ptr(), m1.data_ptr(), B, S, NH, H, 1e-6, cap,
                                             code, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        assert relerr(host(h2), h_ref) < tol and relerr(host(c), st_ref[0]) < tol and relerr(host(n), st_ref[1]) < tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,with_state", [(36, False), (37, False), (197, True), (198, True)])
def test_slstm_scan_single_pass_forms(ops, B, with_state, dtype):
    """Around the numbers of warps at which the single pass changes from one unit a lane to a 16-byte vector."""
    rng = np.random.default_rng(B)
    rnd = xo.bf16_round if dtype == torch.bfloat16 else (lambda a: a)
    S, NH, H = 43, 4, 72
    z = rnd(rng.standard_normal((B, S, NH, H)).astype(np.float32))
    i, f, o = (rnd((rng.standard_normal((B, S, NH)) + s).astype(np.float32)) for s in (0, 3, 0))
    st0 = (rng.standard_normal((B, NH, H)).astype(np.float32), rng.uniform(0.5, 2, (B, NH, H)).astype(np.float32),
           rng.standard_normal((B, NH)).astype(np.float32)) if with_state else None
    h_ref, st_ref = xo.slstm_scan(z, i, f, o, st0)
    h, st1 = ops.slstm_scan(*(dev(a, dtype) for a in (z, i, f, o)), state=None if st0 is None else tuple(dev(s) for s in st0))
    assert relerr(host(h), h_ref) < (FP32_TOL if dtype == torch.float32 else BF16_TOL)
    for a, r in zip(st1, st_ref):
        assert relerr(host(a), r) < FP32_TOL


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("closed", [-1e4, -1e6, -1e9, float(np.finfo(np.float32).min), -np.inf])
def test_slstm_scan_closed_gates(ops, closed, dtype):
    """Tokens that reset the state (a forget gate closed for good) or that are masked out (input gate closed), in the middle and
    at the edges of segments: what lies after them keeps the accuracy of the step-by-step oracle."""
    rng = np.random.default_rng(11)
    rnd = xo.bf16_round if dtype == torch.bfloat16 else (lambda a: a)
    B, S, NH, H = 1, 1024, 2, 128
    z = rnd(rng.standard_normal((B, S, NH, H)).astype(np.float32))
    i, f, o = (rnd((rng.standard_normal((B, S, NH)) + s).astype(np.float32)) for s in (0, 3, 0))
    f[:, [200, 511, 768], 0] = closed
    f[:, 40, 1] = closed
    i[:, 100:180, 1] = closed
    f, i = rnd(f), rnd(i)
    st0 = (rng.standard_normal((B, NH, H)).astype(np.float32), rng.uniform(0.5, 2, (B, NH, H)).astype(np.float32),
           rng.standard_normal((B, NH)).astype(np.float32))
    args = [dev(a, dtype) for a in (z, i, f, o)]
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    for st in (None, st0):
        h_ref, st_ref = xo.slstm_scan(*(host(a) for a in args), st)
        assert np.isfinite(h_ref).all()
        h, st1 = ops.slstm_scan(*args, state=None if st is None else tuple(dev(s) for s in st))
        assert relerr(host(h), h_ref) < tol
        for a, r in zip(st1, st_ref):
            assert relerr(host(a), r) < tol


@pytest.mark.parametrize("S", [4, 1024])
def test_slstm_scan_keeps_small_inputs(ops, S):
    """c is fp32 whatever the activations are: small z (where 1 - 2 / (1 + e^2z) would leave two digits) keep fp32 accuracy."""
    rng = np.random.default_rng(S)
    z = xo.bf16_round((rng.standard_normal((1, S, 2, 64)) * 1e-5).astype(np.float32))
    i, f, o = (xo.bf16_round((rng.standard_normal((1, S, 2)) + s).astype(np.float32)) for s in (0, 3, 0))
    _, st_ref = xo.slstm_scan(z, i, f, o)
    _, st = ops.slstm_scan(*(dev(a, torch.bfloat16) for a in (z, i, f, o)))
    for a, r in zip(st, st_ref):
        assert relerr(host(a), r) < FP32_TOL


def test_slstm_recurrent_fixture(ops, golden):
    g = golden("slstm_b")
    nh = int(g["num_heads"])
    hs, st = ops.slstm_recurrent(dev(g["gx"]), dev(g["R"]), dev(g["rb"]), None, nh, 15.0)
    assert relerr(host(hs), g["hs"]) < FP32_TOL
    for got, key in zip(st, "cnhm"):
        assert relerr(host(got), g[key]) < FP32_TOL
    hs2, st2 = ops.slstm_recurrent(dev(g["gx2"]), dev(g["R"]), dev(g["rb"]), st, nh, 15.0)
    assert relerr(host(hs2), g["hs2"]) < FP32_TOL
    for got, key in zip(st2, ("c2", "n2", "h2", "m2")):
        assert relerr(host(got), g[key]) < FP32_TOL


@pytest.mark.parametrize("B,S,NH,dh,dtype", [(5, 40, 4, 256, torch.float32), (9, 24, 2, 64, torch.float32),
                                              (8, 48, 4, 256, torch.bfloat16), (3, 17, 3, 128, torch.bfloat16)])
def test_slstm_recurrent_oracle(ops, B, S, NH, dh, dtype):
    rng = np.random.default_rng(dh + B)
    rd = xo.bf16_round if dtype == torch.bfloat16 else (lambda a: a)
    D = NH * dh
    gx = rd(rng.standard_normal((B, S, 4, D)).astype(np.float32))
    gx[:, :, 1] += np.linspace(3, 6, D, dtype=np.float32)
    gx = rd(gx)
    R = rd((rng.standard_normal((4, NH, dh, dh)) * 0.02).astype(np.float32))
    rb = (rng.standard_normal((4, D)) * 0.05).astype(np.float32)
    hs_ref, st_ref = xo.slstm_recurrent(gx, R, rb, None, NH, 15.0)
    hs, st = ops.slstm_recurrent(dev(gx, dtype), dev(R, dtype), dev(rb), None, NH, 15.0)
    tol = BF16_TOL if dtype == torch.bfloat16 else FP32_TOL
    assert relerr(host(hs), hs_ref) < tol
    for got, want in zip(st, st_ref):
        assert relerr(host(got), want) < (tol if dtype == torch.bfloat16 else FP32_TOL)


@pytest.mark.parametrize("B,S,NH", [(1, 5, 1), (33, 70, 2), (32, 600, 4)])
def test_slstm_recurrent_tensor_core_path(ops, B, S, NH):
    """bf16 with head dimension 256 runs on the tensor cores (h fed back as bf16): ragged batch groups, a carried
    state, and a long sequence for drift."""
    dh, D = 256, NH * 256
    rng = np.random.default_rng(B * 1000 + S)
    gx = rng.standard_normal((B, S, 4, D)).astype(np.float32)
    gx[:, :, 1] += np.linspace(3, 6, D, dtype=np.float32)
    gx = xo.bf16_round(gx)
    R = xo.bf16_round((rng.standard_normal((4, NH, dh, dh)) * 0.02).astype(np.float32))
    rb = (rng.standard_normal((4, D)) * 0.05).astype(np.float32)
    bf = torch.bfloat16
    S1 = S // 2
    hs_ref, st_ref = xo.slstm_recurrent(gx, R, rb, None, NH, 15.0)
    hs1, st1 = ops.slstm_recurrent(dev(gx[:, :S1], bf), dev(R, bf), dev(rb), None, NH, 15.0)
    hs2, st2 = ops.slstm_recurrent(dev(gx[:, S1:], bf), dev(R, bf), dev(rb), st1, NH, 15.0)
    hs = torch.cat([hs1, hs2], 1)
    assert torch.isfinite(hs.float()).all()
    assert relerr(host(hs), hs_ref) < BF16_TOL
    for got, want in zip(st2, st_ref):
        assert relerr(host(got), want) < BF16_TOL


BF, FP = torch.bfloat16, torch.float32


@pytest.mark.parametrize("B,S,NH,dh,dtype", [(1, 1, 1, 64, BF), (16, 2, 2, 64, BF), (17, 3, 4, 128, BF), (5, 64, 2, 128, BF),
                                             (16, 1, 1, 256, BF), (15, 2, 2, 256, BF), (34, 7, 3, 256, BF),
                                             (8, 3, 2, 64, BF), (9, 3, 1, 128, BF), (7, 4, 1, 256, BF),
                                             (209, 4, 4, 256, BF), (139, 3, 8, 128, BF), (265, 2, 8, 64, BF),
                                             (1, 1, 1, 256, FP), (4, 2, 2, 128, FP), (5, 3, 2, 64, FP), (33, 40, 4, 256, FP),
                                             (70, 5, 4, 128, FP), (140, 4, 4, 64, FP)])
def test_slstm_recurrent_edges(ops, B, S, NH, dh, dtype):
    """One, two and three steps (each h buffer unused, used once, reused), rows around the groups of a cluster (8 in bf16, 16
    where those would not be resident at once, 4 in fp32), a carried state.  bf16 heads of 64 and 128 feed h back unrounded and use the exact exponentials: their states stay within
    the fp32 tolerance and their outputs within half a bf16 ulp (8 significant bits: 2^-8 of the value) of it."""
    rng = np.random.default_rng(dh + B)
    rd = xo.bf16_round if dtype == BF else (lambda a: a)
    D = NH * dh
    gx = rng.standard_normal((B, S, 4, D)).astype(np.float32)
    gx[:, :, 1] += np.linspace(3, 6, D, dtype=np.float32)
    gx = rd(gx)
    R = rd((rng.standard_normal((4, NH, dh, dh)) * 0.05).astype(np.float32))
    rb = (rng.standard_normal((4, D)) * 0.05).astype(np.float32)
    st0 = [rng.standard_normal((B, D)).astype(np.float32) for _ in range(4)]
    st0[1] = np.abs(st0[1]) + 1
    hs_ref, st_ref = xo.slstm_recurrent(gx, R, rb, tuple(st0), NH, 15.0)
    hs, st = ops.slstm_recurrent(dev(gx, dtype), dev(R, dtype), dev(rb), tuple(dev(s) for s in st0), NH, 15.0)
    ops.slstm_recurrent_status()
    rounded = dtype == BF and dh == 256
    for got, want in zip(st, st_ref):
        assert relerr(host(got), want) < (BF16_TOL if rounded else FP32_TOL)
    assert relerr(host(hs), hs_ref) < (BF16_TOL if rounded else FP32_TOL if dtype == FP else 2.0 ** -8 + FP32_TOL)


@pytest.mark.parametrize("dh,dtype", [(64, BF), (128, BF), (256, BF), (64, FP), (128, FP), (256, FP), (32, FP)])
@pytest.mark.parametrize("cap", [15.0, 0.0])
def test_slstm_recurrent_keeps_nan_and_inf(ops, dh, dtype, cap):
    """A NaN in any gate's pre-activation reaches the same outputs and states as in the oracle; an infinite cell input or
    output gate saturates."""
    B, S, NH = 5, 2, 1
    rng = np.random.default_rng(dh)
    rd = xo.bf16_round if dtype == BF else (lambda a: a)
    gx = rd(rng.standard_normal((B, S, 4, dh)).astype(np.float32))
    for g in range(4):
        gx[g, 0, g, 3 + g] = np.nan
    gx[4, 0, 2, 5], gx[4, 1, 2, 6], gx[4, 0, 3, 7], gx[4, 1, 3, 8] = np.inf, -np.inf, np.inf, -np.inf
    R = rd((rng.standard_normal((4, NH, dh, dh)) * 0.05).astype(np.float32))
    rb = np.zeros((4, dh), np.float32)
    hs_ref, st_ref = xo.slstm_recurrent(gx, R, rb, None, NH, cap)
    hs, st = ops.slstm_recurrent(dev(gx, dtype), dev(R, dtype), dev(rb), None, NH, cap)
    ops.slstm_recurrent_status()
    for got, want in zip((hs, *st), (hs_ref, *st_ref)):
        got = host(got)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert relerr(np.nan_to_num(got), np.nan_to_num(want)) < BF16_TOL


def test_front_end_refuses_sizes_that_do_not_fit(ops):
    """The ABI takes bare pointers, so operands that are too small, of another dtype or incomplete are refused before a launch."""
    z = lambda *s, dt=torch.bfloat16: torch.zeros(*s, device="cuda", dtype=dt)
    B, NH, dqk, dv, S = 2, 2, 16, 32, 8
    f32 = torch.float32
    st = (z(B, NH, dqk, dv, dt=f32), z(B, NH, dqk, dt=f32), z(B, NH, dt=f32))
    step = dict(q=z(B, NH, dqk), k=z(B, NH, dqk), v=z(B, NH, dv), i=z(B, NH), f=z(B, NH), state=st)
    gated = dict(step, ogate=z(B, NH * dv), norm_weight=z(NH * dv))
    chunk = dict(q=z(B, NH, S, dqk), k=z(B, NH, S, dqk), v=z(B, NH, S, dv), i=z(B, NH, S), f=z(B, NH, S), state=st)
    lin = dict(weight=z(64, 32), x=z(3, 32), bias=z(64), residual=z(3, 64))
    small = [(ops.mlstm_step, step, dict(k=z(B, NH, 8))), (ops.mlstm_step, step, dict(v=z(1, NH, dv))),
             (ops.mlstm_step, step, dict(f=z(B, 1))), (ops.mlstm_step, step, dict(state=(st[0][:1], st[1], st[2]))),
             (ops.mlstm_step, step, dict(state=(st[0], st[1][:1], st[2]))), (ops.mlstm_step, step, dict(state=(st[0], None, None))),
             (ops.mlstm_step, step, dict(state=(None, st[1], st[2]))),
             (ops.mlstm_step_gated, gated, dict(k=z(B, NH, 8))), (ops.mlstm_step_gated, gated, dict(ogate=z(1, NH * dv))),
             (ops.mlstm_step_gated, gated, dict(norm_weight=z(dv))), (ops.mlstm_step_gated, gated, dict(i=z(1, NH))),
             (ops.mlstm_chunkwise, chunk, dict(k=z(B, NH, S, 8))), (ops.mlstm_chunkwise, chunk, dict(v=z(B, NH, 4, dv))),
             (ops.mlstm_chunkwise, chunk, dict(i=z(B, NH, 4), f=z(B, NH, 4))),
             (ops.mlstm_chunkwise, chunk, dict(state=(st[0], st[1][:1], st[2])))]
    for fn in (ops.linear_token, ops.linear_rows):
        small += [(fn, lin, dict(weight=z(64, 16))), (fn, lin, dict(bias=z(32))), (fn, lin, dict(residual=z(2, 64))),
                  (fn, lin, dict(weight=z(63, 32), bias=None, residual=None, swiglu_pair=True))]
    small += [(ops.rms_norm, dict(x=z(4, 64), weight=z(32), eps=1e-6), {}),
              (ops.add_rms_norm, dict(x=z(4, 64), residual=z(3, 64), weight=z(64)), {})]
    for fn, good, bad in small:
        with pytest.raises(ValueError):
            fn(**dict(good, **bad))
    for bad in (dict(k=z(B, NH, dqk, dt=f32)), dict(v=z(B, NH, dv, dt=f32))):
        with pytest.raises(TypeError):
            ops.mlstm_step(**dict(step, **bad))
        with pytest.raises(TypeError):
            ops.mlstm_step_gated(**dict(gated, **bad))
    with pytest.raises((ValueError, TypeError)):
        ops.mlstm_step(**dict(step, state=()))
    for fn, good in ((ops.mlstm_step, step), (ops.mlstm_step_gated, gated), (ops.mlstm_chunkwise, chunk), (ops.linear_rows, lin)):
        fn(**good)


def test_front_end_releases_the_interpreter_lock(ops):
    """Other Python threads run while a launch is on its way (as through ctypes): with thread switching on request put off for
    good, a waiting thread can only get the lock where a call gives it up."""
    import threading
    x = torch.zeros(4, 64, device="cuda")
    ops.rms_norm(x, None)
    go, ran, interval = threading.Lock(), [], sys.getswitchinterval()
    go.acquire()
    other = threading.Thread(target=lambda: (go.acquire(), ran.append(True)))
    other.start()
    kept = []                    # (freeing a tensor gives the lock up as well)
    try:
        sys.setswitchinterval(1e3)
        go.release()
        while not ran and len(kept) < 20000:
            kept.append(ops.rms_norm(x, None))
    finally:
        sys.setswitchinterval(interval)
        other.join()
    assert len(kept) < 20000


def test_step_with_an_unaligned_v(ops):
    """v is read four elements at a time: a view at an odd offset is copied, in the plain and in the gated step."""
    torch.manual_seed(0)
    B, NH, dqk, dv = 2, 2, 16, 32
    for dt in (torch.float32, torch.bfloat16):
        q, k = (torch.randn(B, NH, dqk, device="cuda").to(dt) for _ in range(2))
        v = torch.randn(B * NH * dv + 1, device="cuda").to(dt)[1:].view(B, NH, dv)
        i, f, og = (torch.randn(*s, device="cuda").to(dt) for s in ((B, NH), (B, NH), (B, NH * dv)))
        assert torch.equal(ops.mlstm_step(q, k, v, i, f)[0], ops.mlstm_step(q, k, v.clone(), i, f)[0])
        assert torch.equal(ops.mlstm_step_gated(q, k, v, i, f, og, None)[0],
                           ops.mlstm_step_gated(q, k, v.clone(), i.reshape(-1), f.unsqueeze(-1), og, None)[0])
    from xlstm_cuda import _lib
    C = torch.zeros(B * NH * dqk * dv + 1, device="cuda")[1:].view(B, NH, dqk, dv)
    with pytest.raises(_lib.XlstmCudaError):
        ops.mlstm_step(q, k, v.clone(), i, f, (C, torch.zeros(B, NH, dqk, device="cuda"), torch.zeros(B, NH, device="cuda")))


@pytest.mark.parametrize("state_dtype,strided", [(torch.bfloat16, False), (torch.float32, True)])
def test_step_with_a_state_that_is_converted(ops, state_dtype, strided):
    """A state in bf16 or with strides is copied by the launch right before the step: it is not read early, also where the
    caller vouches for the state that it passes."""
    torch.manual_seed(1)
    B, NH, dqk, dv = 16, 8, 256, 512
    bf = torch.bfloat16
    q, k = (torch.randn(B, NH, dqk, device="cuda").to(bf) for _ in range(2))
    v = torch.randn(B, NH, dv, device="cuda").to(bf)
    i, f, og = (torch.randn(*s, device="cuda").to(bf) for s in ((B, NH), (B, NH), (B, NH * dv)))
    w = torch.ones(NH * dv, device="cuda", dtype=bf)
    n, m = torch.randn(B, NH, dqk, device="cuda"), torch.zeros(B, NH, device="cuda")
    for _ in range(20):
        C = torch.randn(B, NH, dqk, dv, device="cuda").to(state_dtype)
        given = C.transpose(2, 3).contiguous().transpose(2, 3) if strided else C
        h, (C1, _, _) = ops.mlstm_step(q, k, v, i, f, (C.float(), n, m))
        h2, (C2, _, _) = ops.mlstm_step(q, k, v, i, f, (given, n, m), state_settled=True)
        assert torch.equal(h, h2) and torch.equal(C1, C2)
        y, _ = ops.mlstm_step_gated(q, k, v, i, f, og, w, (C.float(), n, m))
        y2, _ = ops.mlstm_step_gated(q, k, v, i, f, og, w, (given, n, m), state_settled=True)
        assert torch.equal(y, y2)


@pytest.mark.parametrize("part", ["n", "m"])
@pytest.mark.parametrize("form", ["bf16", "strided", "written"])
@pytest.mark.parametrize("B,dqk,dv", [(1, 256, 512), (16, 256, 512)])
def test_step_with_a_normaliser_or_stabiliser_written_just_before(ops, part, form, B, dqk, dv):
    """A settled state vouches for C alone.  n or m in bf16 or with strides is copied by the launch right before the step, or the
    caller writes it there: the step sees what was written, bit for bit, through the plain step, the gated one and a block's token."""
    from xlstm_cuda.blocks import mLSTMBlock
    torch.manual_seed(2)
    NH, bf = 8, torch.bfloat16
    rnd = lambda *s: torch.randn(*s, device="cuda")
    q, k, v = rnd(B, NH, dqk).to(bf), rnd(B, NH, dqk).to(bf), rnd(B, NH, dv).to(bf)
    i, f, og = rnd(B, NH).to(bf), rnd(B, NH).to(bf), rnd(B, NH * dv).to(bf)
    w = torch.ones(NH * dv, device="cuda", dtype=bf)
    with torch.inference_mode():
        blk = mLSTMBlock(0, embedding_dim=512, num_heads=4, compute_dtype=bf).cuda().to(bf)
        blk.fuse_projections()
        cell = blk.mlstm_cell
        bh, bk, bv = cell.num_heads, cell.qk_dim_per_head, cell.v_dim_per_head
        x = rnd(B, 1, 512).to(bf)

        def states(shape_heads, dk, dvv):
            """(what the step is given, the same values settled long ago)"""
            C, n, m = rnd(B, shape_heads, dk, dvv), rnd(B, shape_heads, dk), rnd(B, shape_heads)
            src = n if part == "n" else m
            if form == "bf16":
                src.copy_(src.to(bf))
            plain = (C, n.clone(), m.clone())
            if form == "bf16":
                given = src.to(bf)
            elif form == "strided":
                given = torch.stack([src, src], -1)[..., 0]
            else:
                given = torch.full_like(src, 7.0)
            torch.cuda.synchronize()

            def write():
                if form == "written":
                    given.copy_(src)
            return ((C, given, m) if part == "n" else (C, n, given)), plain, write

        for _ in range(10):
            st, plain, write = states(NH, dqk, dv)
            ref = ops.mlstm_step(q, k, v, i, f, plain)
            write()
            got = ops.mlstm_step(q, k, v, i, f, st, state_settled=True)
            for a, b in zip((got[0], *got[1]), (ref[0], *ref[1])):
                assert torch.equal(a, b)
            st, plain, write = states(NH, dqk, dv)
            ref = ops.mlstm_step_gated(q, k, v, i, f, og, w, plain)
            write()
            got = ops.mlstm_step_gated(q, k, v, i, f, og, w, st, state_settled=True)
            for a, b in zip((got[0], *got[1]), (ref[0], *ref[1])):
                assert torch.equal(a, b)
            st, plain, write = states(bh, bk, bv)
            ref = blk(x, plain)
            write()
            got = blk(x, st)
            for a, b in zip((got[0], *got[1]), (ref[0], *ref[1])):
                assert torch.equal(a, b)


# ---- error behaviour of the C ABI --------------------------------------------------
def test_errors_are_statuses_not_crashes(ops):
    from xlstm_cuda import _lib
    lib = _lib.load()
    assert lib.xlstm_softcap(None, None, 8, 15.0, 0, None) == -1
    assert lib.xlstm_softcap(None, None, 0, 15.0, 0, None) == 0
    x = torch.zeros(16, device="cuda")
    assert lib.xlstm_softcap(x.data_ptr(), x.data_ptr(), 16, 15.0, 7, None) == -2
    assert lib.xlstm_mlstm_step(*([x.data_ptr()] * 5), None, None, None, *([x.data_ptr()] * 4), 1, 1, 2, 3, 1e-6, 0, None) == -2
    px = x.data_ptr()
    # flags the step does not know: invalid; output epilogue wider than eight 64-column tiles: unsupported (no launch)
    assert lib.xlstm_mlstm_step_ex(*([px] * 5), None, None, None, *([px] * 4), 1, 1, 8, 8, 1e-6, 0.0, 2, 0, None) == -1
    assert lib.xlstm_mlstm_step_gated(*([px] * 5), None, None, None, px, 1024, None, 1e-6, *([px] * 4), 1, 1, 8, 1024, 1e-6, 0.0,
                                      0, 0, None) == -2
    assert lib.xlstm_mlstm_step_gated(*([px] * 5), None, None, None, None, 8, None, 1e-6, *([px] * 4), 1, 1, 8, 8, 1e-6, 0.0,
                                      0, 0, None) == -1
    with pytest.raises(RuntimeError):
        ops.softcap(torch.zeros(4), 15.0)  # CPU tensor: no fallback
    with pytest.raises(TypeError):
        ops.softcap(torch.zeros(4, device="cuda", dtype=torch.float16), 15.0)


# ---- gate soft-cap folded into the kernels -------------------------------------------------
@pytest.mark.parametrize("dtype,shape", [(torch.float32, (2, 3, 200, 64, 64)), (torch.bfloat16, (2, 2, 300, 256, 256))])
def test_gate_cap_inside_the_kernels(ops, dtype, shape):
    """Raw gate projections + gate_cap give what pre-capped gates give: chunkwise (exact path in
    fp32, tensor-core path + exact tail in bf16) and the decode step."""
    B, NH, S, dqk, dv = shape
    rng = np.random.default_rng(S)
    q, k = (rng.standard_normal((B, NH, S, dqk)).astype(np.float32) for _ in range(2))
    v = rng.standard_normal((B, NH, S, dv)).astype(np.float32)
    i_raw = (rng.standard_normal((B, NH, S)) * 6.0).astype(np.float32)        # well into the tanh knee
    f_raw = (rng.standard_normal((B, NH, S)) * 6.0 + 8.0).astype(np.float32)
    if dtype == torch.bfloat16:
        q, k, v, i_raw, f_raw = (xo.bf16_round(a) for a in (q, k, v, i_raw, f_raw))
    cap = 15.0
    i_cap, f_cap = xo.softcap(i_raw, cap), xo.softcap(f_raw, cap)
    h_ref, (C_ref, n_ref, m_ref) = xo.mlstm_recurrent(q, k, v, i_cap, f_cap, None, 1e-6)
    tol = FP32_TOL if dtype == torch.float32 else BF16_TOL
    h, (C, n, m) = ops.mlstm_chunkwise(dev(q, dtype), dev(k, dtype), dev(v, dtype), dev(i_raw, dtype), dev(f_raw, dtype),
                                       None, 64, 1e-6, gate_cap=cap)
    assert relerr(host(h), h_ref) <= tol and relerr(host(C), C_ref) <= tol and relerr(host(n), n_ref) <= tol
    assert np.abs(host(m) - m_ref).max() <= (1e-4 if dtype == torch.float32 else 2e-2)
    # decode steps from that state, raw gates again
    st, st_ref = (C, n, m), (C_ref, n_ref, m_ref)
    for t in range(3):
        qs, ks, vs = q[:, :, t], k[:, :, t], v[:, :, t]
        hs, st = ops.mlstm_step(dev(qs, dtype), dev(ks, dtype), dev(vs, dtype), dev(i_raw[:, :, t], dtype),
                                dev(f_raw[:, :, t], dtype), st, 1e-6, gate_cap=cap)
        hr, st_ref = xo.mlstm_recurrent(qs[:, :, None], ks[:, :, None], vs[:, :, None], i_cap[:, :, t:t + 1],
                                        f_cap[:, :, t:t + 1], st_ref, 1e-6)
        assert relerr(host(hs), hr[:, :, 0]) <= tol
    # cap <= 0 / None: gates are taken as given
    h0, _ = ops.mlstm_chunkwise(dev(q, dtype), dev(k, dtype), dev(v, dtype), dev(i_cap, dtype), dev(f_cap, dtype), None, 64, 1e-6)
    h1, _ = ops.mlstm_chunkwise(dev(q, dtype), dev(k, dtype), dev(v, dtype), dev(i_cap, dtype), dev(f_cap, dtype), None, 64, 1e-6,
                                gate_cap=0.0)
    assert torch.equal(h0, h1)


@pytest.mark.parametrize("S", [128 + 1, 128 + 64, 128 + 65, 128 + 127, 128 + 128])
def test_chunkwise_tail_forms(ops, S):
    """One tile and a tail of any length against the oracle, and with scratch for the tile alone: a tail needs none, so a caller who
    has sized it so gets the same, and two tiles are refused."""
    rng = np.random.default_rng(S)
    NH, dqk, dv = 2, 128, 256
    q, k = (xo.bf16_round(rng.standard_normal((1, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = xo.bf16_round(rng.standard_normal((1, NH, S, dv)).astype(np.float32))
    i, f = (xo.bf16_round(a) for a in gates(rng, (1, NH, S)))
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f)
    args = [dev(a, torch.bfloat16) for a in (q, k, v, i, f)]
    h, st = ops.mlstm_chunkwise(*args)
    assert relerr(host(h), h_ref) < BF16_TOL
    for a, r in zip(st, st_ref):
        assert relerr(host(a), r) < BF16_TOL
    from xlstm_cuda import _lib
    least = _lib.load().xlstm_mlstm_chunkwise_workspace_bytes(1, NH, 128, dqk, dv, 64, _lib.BF16)   # one tile, no tail
    ws = torch.empty(least, dtype=torch.uint8, device="cuda")
    C, n, m = torch.empty_like(st[0]), torch.empty_like(st[1]), torch.empty_like(st[2])
    h2 = torch.empty_like(h)
    rc = _lib.load().xlstm_mlstm_chunkwise_fwd(*(a.data_ptr() for a in args), None, None, None, h2.data_ptr(), C.data_ptr(), n.data_ptr(),
                                               m.data_ptr(), 1, NH, S, dqk, dv, 64, 1e-6, _lib.BF16, None, ws.data_ptr(), least,
                                               torch.cuda.current_stream().cuda_stream)
    assert (rc == 0) == (S < 256)        # 256 tokens are two tiles
    if rc == 0:
        assert relerr(host(h2)[:, :, 128:], host(h)[:, :, 128:]) < 2.0 ** -7 + FP32_TOL
        assert relerr(host(C), host(st[0])) < FP32_TOL


@pytest.mark.parametrize("tail", [1, 63, 64, 65, 127])
@pytest.mark.parametrize("NH,dqk,dv,f_mean", [(3, 256, 512, 3.0), (3, 128, 256, -7.0), (12, 256, 512, -7.0), (40, 128, 256, 3.0)])
def test_chunkwise_tail_behind_tiles_equals_fp32_from_their_state(ops, tail, NH, dqk, dv, f_mean):
    """The tokens behind two tensor-core tiles, of bounded and of widely spread gates, for fewer and more CTAs than SMs: the state
    within 1e-5 of the fp32 kernels' from the state that the tiles alone leave, h within one bf16 rounding (2^-8 of the value) and
    1e-4 of the row on rows whose normaliser does not cancel."""
    torch.manual_seed(tail + NH)
    S = 256 + tail
    q, k, v = (torch.randn(1, NH, S, d, device="cuda").to(BF) for d in (dqk, dqk, dv))
    i, f = torch.randn(1, NH, S, device="cuda").to(BF), (torch.randn(1, NH, S, device="cuda") + f_mean).to(BF)
    cut = lambda a, b: [x[:, :, a:b] for x in (q, k, v, i, f)]
    try:
        ops.chunkwise_segments(1)
        h, st = ops.mlstm_chunkwise(*cut(0, S))
        _, mid = ops.mlstm_chunkwise(*cut(0, 256))
    finally:
        ops.chunkwise_segments(None)
    hf, sf = ops.mlstm_chunkwise(*(x.float() for x in cut(256, S)), mid)
    for a, b in zip(st, sf):
        assert relerr(host(a), host(b)) < 1e-5
    qs, n = q[:, :, 256:].double() / dqk ** 0.5, []
    nn, m = mid[1].double(), mid[2].double()
    for t in range(256, S):
        fl, it = torch.nn.functional.logsigmoid(f[:, :, t].double()), i[:, :, t].double()
        mn = torch.maximum(fl + m, it)
        nn = torch.exp(fl + m - mn)[..., None] * nn + torch.exp(it - mn)[..., None] * k[:, :, t].double()
        m = mn
        n.append((nn, torch.exp(-m)))
    den = torch.stack([torch.maximum((qs[:, :, j] * a).sum(-1).abs(), e) for j, (a, e) in enumerate(n)], 2)
    cond = qs.norm(dim=-1) * torch.stack([a.norm(dim=-1) for a, _ in n], 2) / den
    off = (h[:, :, 256:].double() - hf.double()).abs()
    room = 2.0 ** -8 * hf.double().abs() + 1e-4 * hf.double().abs().amax(-1, keepdim=True)
    assert bool(((off <= room) | (cond >= 20)[..., None]).all())


@pytest.mark.parametrize("T", [2, 15, 16, 17, 33, 63, 64, 65, 96, 97, 127])
@pytest.mark.parametrize("dqk,dv,state,f_mean", [(256, 512, True, 3.0), (256, 128, False, -2.0), (128, 96, True, 6.0), (128, 256, False, 3.0)])
def test_chunkwise_short_bf16(ops, T, dqk, dv, state, f_mean):
    """Fewer tokens than a tensor-core tile, to fp32 accuracy in one launch: sizes around the 16-token blocks, the 32-token
    passes and the two tile sizes, without and with a state, from strided q, k, v.  States within 1e-5 of the float64 recurrence
    (sums of up to 127 products in fp32), h within that and one bf16 rounding (2^-8 of the value) on rows whose normaliser does
    not cancel, and as near to float64 as the fp32 kernels are."""
    rng = np.random.default_rng(T * 7 + dqk + dv)
    B, NH = 2, 3
    rd = xo.bf16_round
    q, k = (rd(rng.standard_normal((B, NH, T, dqk)).astype(np.float32)) for _ in range(2))
    v = rd(rng.standard_normal((B, NH, T, dv)).astype(np.float32))
    i = rd(rng.standard_normal((B, NH, T)).astype(np.float32))
    f = rd((rng.standard_normal((B, NH, T)) + f_mean).astype(np.float32))
    st0 = None
    if state:
        st0 = (rng.standard_normal((B, NH, dqk, dv)).astype(np.float32), rng.standard_normal((B, NH, dqk)).astype(np.float32),
               rng.standard_normal((B, NH)).astype(np.float32))
    C, n, m = (np.zeros((B, NH, dqk, dv)), np.zeros((B, NH, dqk)), np.zeros((B, NH))) if st0 is None else (a.astype(np.float64) for a in st0)
    h64, cond = [], []
    for t in range(T):
        fl = -np.logaddexp(0, -f[:, :, t].astype(np.float64))
        mn = np.maximum(fl + m, i[:, :, t])
        fg, ig = np.exp(fl + m - mn), np.exp(i[:, :, t] - mn)
        C = fg[..., None, None] * C + ig[..., None, None] * k[:, :, t, :, None].astype(np.float64) * v[:, :, t, None, :]
        n = fg[..., None] * n + ig[..., None] * k[:, :, t]
        m = mn
        qs = q[:, :, t].astype(np.float64) / np.sqrt(dqk)
        qn = np.einsum("bhd,bhd->bh", qs, n)
        den = np.maximum(np.abs(qn), np.exp(-m)) + 1e-6
        h64.append(np.einsum("bhd,bhdv->bhv", qs, C) / den[..., None])
        cond.append(np.linalg.norm(qs, axis=-1) * np.linalg.norm(n, axis=-1) / den)
    h64, cond = np.stack(h64, 2), np.stack(cond, 2)
    # q and k as column blocks of one wider projection, token-major
    qk = dev(np.concatenate([q, k], -1), BF).permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    args = (qk[..., :dqk], qk[..., dqk:], dev(v, BF).permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3), dev(i, BF), dev(f, BF))
    h, st = ops.mlstm_chunkwise(*args, None if st0 is None else tuple(dev(s) for s in st0))
    hf, stf = ops.mlstm_chunkwise(*(dev(a) for a in (q, k, v, i, f)), None if st0 is None else tuple(dev(s) for s in st0))
    for got, f32, want in zip(st, stf, (C, n, m)):
        e = relerr(host(got), want)
        assert e < 1e-5 and e <= 2 * relerr(host(f32), want) + 3e-7
    ok = (cond < 20)[..., None]
    off = np.abs(host(h) - h64) * ok
    assert (off <= 2.0 ** -8 * np.abs(h64) + 1e-4 * np.abs(h64 * ok).max()).all()
    if not state:   # a carried state equals the sequence that made it
        h2, st2 = ops.mlstm_chunkwise(*(a[:, :, :1 + T // 2] for a in args), None)
        if T - (1 + T // 2) > 0:
            h3, st3 = ops.mlstm_chunkwise(*(a[:, :, 1 + T // 2:] for a in args), st2)
            for got, want in zip(st3, st):
                assert relerr(host(got), host(want)) < 1e-5


@pytest.mark.parametrize("T", [20, 30, 60, 100, 127])
@pytest.mark.parametrize("dqk,dv", [(256, 512), (128, 96)])
def test_chunkwise_short_bf16_keeps_an_infinity_to_later_tokens(ops, T, dqk, dv):
    """An infinite v reaches its own column of its block of 16 tokens and of those after it, as in the fp32 kernels: the blocks
    before it and the other columns of h are bit for bit what they are without it, those of C to fp32 rounding (their sums go
    without the grids then)."""
    torch.manual_seed(T + dqk)
    q, k, v = (torch.randn(1, 2, T, d, device="cuda").to(BF) for d in (dqk, dqk, dv))
    i, f = torch.randn(1, 2, T, device="cuda").to(BF), (torch.randn(1, 2, T, device="cuda") + 3).to(BF)
    st = (torch.randn(1, 2, dqk, dv, device="cuda"), torch.randn(1, 2, dqk, device="cuda"), torch.zeros(1, 2, device="cuda"))
    h, (C, n, m) = ops.mlstm_chunkwise(q, k, v, i, f, st)
    for at in (17, T - 1):
        vi = v.clone()
        vi[:, :, at, 5] = float("inf")
        hi, (Ci, ni, mi) = ops.mlstm_chunkwise(q, k, vi, i, f, st)
        assert torch.equal(hi[:, :, :at // 16 * 16], h[:, :, :at // 16 * 16])
        others = torch.arange(dv, device="cuda") != 5
        assert torch.equal(hi[..., others], h[..., others]) and torch.equal(ni, n) and torch.equal(mi, m)
        assert not torch.isfinite(hi[:, :, at:, 5].float()).any()
        assert (Ci[..., 5][k[:, :, at] != 0].isinf()).all() and relerr(host(Ci[..., others]), host(C[..., others])) < 1e-6


@pytest.mark.parametrize("T", [65, 80, 127, 128])
@pytest.mark.parametrize("dqk,dv,NH,f_mean", [(256, 480, 10, -2.0), (256, 480, 10, 3.0), (128, 96, 50, 3.0)])
def test_chunkwise_short_bf16_in_turn(ops, T, dqk, dv, NH, f_mean):
    """More heads than SMs: 64 tokens at a time in one launch.  As two calls, the second from the first one's state: h to one bf16
    rounding (2^-7 of the value across a rounding boundary) on rows whose normaliser does not cancel, the state to fp32 rounding;
    and no further from float64 than the fp32 kernels (as above)."""
    torch.manual_seed(T + dqk)
    rnd = lambda *s: torch.randn(*s, device="cuda")
    q, k, v = rnd(1, NH, T, dqk).to(BF), rnd(1, NH, T, dqk).to(BF), rnd(1, NH, T, dv).to(BF)
    i, f = rnd(1, NH, T).to(BF), (rnd(1, NH, T) + f_mean).to(BF)
    st = (rnd(1, NH, dqk, dv), rnd(1, NH, dqk), rnd(1, NH))
    part = lambda a, b: [x[:, :, a:b] for x in (q, k, v, i, f)]
    for start in (st, None):
        h, s1 = ops.mlstm_chunkwise(*part(0, T), start)
        ha, sa = ops.mlstm_chunkwise(*part(0, 64), start)
        hb, sb = ops.mlstm_chunkwise(*part(64, T), sa)
        assert torch.equal(h[:, :, :64], ha)
        off = (h[:, :, 64:].float() - hb.float()).abs()
        assert float((off > 2.0 ** -7 * hb.float().abs() + 1e-5 * hb.float().abs().amax(-1, keepdim=True)).float().mean()) < 1e-3
        for a, b in zip(s1, sb):
            assert relerr(host(a), host(b)) < 1e-6
    C, m = st[0].double(), st[2].double()
    for t in range(T):
        fl, it = torch.nn.functional.logsigmoid(f[:, :, t].double()), i[:, :, t].double()
        mn = torch.maximum(fl + m, it)
        fg, ig = torch.exp(fl + m - mn), torch.exp(it - mn)
        C = fg[..., None, None] * C + ig[..., None, None] * k[:, :, t, :, None].double() * v[:, :, t, None, :].double()
        m = mn
    (Cb, Cf) = (ops.mlstm_chunkwise(*args, st)[1][0].double() for args in (part(0, T), [x.float() for x in part(0, T)]))
    assert float((Cb - C).norm()) <= 1.1 * float((Cf - C).norm())


@pytest.mark.parametrize("T", [1, 2, 3, 8, 16, 17, 24, 25, 33, 64, 65, 127])
@pytest.mark.parametrize("dqk,dv,f_mean", [(256, 512, -2.0), (256, 512, 3.0), (128, 256, -2.0)])
def test_chunkwise_short_bf16_state_is_no_further_off_than_fp32(ops, T, dqk, dv, f_mean):
    """The state after up to 127 bf16 tokens against float64, beside the same values through the fp32 multiply-adds (2-norms over
    2 dqk dv elements, so equal errors agree to a few percent: 1.1), from a carried state; gates that forget within a few tokens
    leave single roundings to see (3e-8), where the tensor cores' cut-off sums were 6e-8 off."""
    g = torch.Generator(device="cuda").manual_seed(T * 3 + dqk)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k, v = rnd(1, 2, T, dqk).to(BF), rnd(1, 2, T, dqk).to(BF), rnd(1, 2, T, dv).to(BF)
    i, f = rnd(1, 2, T).to(BF), (rnd(1, 2, T) + f_mean).to(BF)
    st = (rnd(1, 2, dqk, dv), rnd(1, 2, dqk), rnd(1, 2))
    C, n, m = (s.double() for s in st)
    for t in range(T):
        fl, it = torch.nn.functional.logsigmoid(f[:, :, t].double()), i[:, :, t].double()
        mn = torch.maximum(fl + m, it)
        fg, ig = torch.exp(fl + m - mn), torch.exp(it - mn)
        C = fg[..., None, None] * C + ig[..., None, None] * k[:, :, t, :, None].double() * v[:, :, t, None, :].double()
        m = mn
    _, (Cb, _, _) = ops.mlstm_chunkwise(q, k, v, i, f, st)
    _, (Cf, _, _) = ops.mlstm_chunkwise(*(a.float() for a in (q, k, v, i, f)), st)
    eb, ef = (float((a.double() - C).norm() / C.norm()) for a in (Cb, Cf))
    assert eb <= 1.1 * ef, (eb, ef)


@pytest.mark.parametrize("shape,f_mean", [((2, 8, 3968, 256, 512), -2.0), ((2, 8, 3968, 256, 512), 3.0), ((1, 4, 2048, 128, 256), -2.0)])
def test_chunkwise_is_deterministic(ops, shape, f_mean):
    """The same call gives the same bits, in the general path (gates that forget within a few tokens) and the bounded one, call
    after call without a wait between them.  A row of Q scaled in place before the last warp had taken its part of q . n showed
    as single elements of h, in one call of twelve at the first shape."""
    B, NH, S, dqk, dv = shape
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    args = [rnd(B, NH, S, dqk).to(BF), rnd(B, NH, S, dqk).to(BF), rnd(B, NH, S, dv).to(BF), rnd(B, NH, S).to(BF),
            (rnd(B, NH, S) + f_mean).to(BF)]
    try:
        ops.chunkwise_segments(1)
        first = ops.mlstm_chunkwise(*args)
        for _ in range(20):
            for h, st in [ops.mlstm_chunkwise(*args) for _ in range(6)]:
                assert torch.equal(h, first[0]) and all(torch.equal(a, b) for a, b in zip(st, first[1]))
    finally:
        ops.chunkwise_segments(None)


@pytest.mark.parametrize("dqk,dv", [(256, 512), (128, 128)])
@pytest.mark.parametrize("f_shift", [0.0, -8.0])
def test_chunkwise_half_columns_equal_whole_ones(ops, dqk, dv, f_shift):
    """Few heads run on CTAs of 64 columns, many on CTAs of 128: a head's results do not depend on how many others there are,
    bit for bit, in both tensor-core paths, with a carried state and an uneven last tile."""
    rng = np.random.default_rng(dqk)
    few, many, S = 1, 40 * 512 // dv, 300
    q, k = (dev(rng.standard_normal((1, many, S, dqk)), BF) for _ in range(2))
    v = dev(rng.standard_normal((1, many, S, dv)), BF)
    i, f = (dev(a, BF) for a in gates(rng, (1, many, S)))
    f = f + f_shift
    st = tuple(dev(rng.standard_normal(s) * 0.1) for s in ((1, many, dqk, dv), (1, many, dqk), (1, many)))
    try:
        ops.chunkwise_segments(1)
        h, s1 = ops.mlstm_chunkwise(q, k, v, i, f, st)
        hf, sf = ops.mlstm_chunkwise(*(a[:, :few] for a in (q, k, v, i, f)), tuple(s[:, :few].contiguous() for s in st))
        assert torch.equal(h[:, :few], hf)
        for a, b in zip(s1, sf):
            assert torch.equal(a[:, :few], b)
        ops.chunkwise_segments(2)   # segments, whose second pass may be narrow
        hp, sp = ops.mlstm_chunkwise(*(a[:, :few] for a in (q, k, v, i, f)), tuple(s[:, :few].contiguous() for s in st))
        assert relerr(host(hp), host(hf)) < BF16_TOL and relerr(host(sp[0]), host(sf[0])) < 1e-3
    finally:
        ops.chunkwise_segments(None)


@pytest.mark.parametrize("B,NH,S,dqk,dv,P", [(2, 9, 300, 256, 512, 1), (2, 20, 256, 256, 512, 1), (1, 40, 133, 128, 256, 1),
                                             (1, 3, 33 * 128 + 5, 128, 256, 1), (1, 5, 9 * 128 + 70, 128, 256, 4)])
def test_chunkwise_heads_of_both_kinds_equal_each_on_its_own(ops, B, NH, S, dqk, dv, P):
    """The two launches run side by side, in the order that the number of CTAs and tiles asks for: up to one CTA per SM (of half
    the columns), more than that, a long pass, segments.  Heads do not depend on one another, so every head gives bit for bit what
    it gives in a call of its own, where only its kind runs (few CTAs, general launch first)."""
    rng = np.random.default_rng(NH * S)
    q, k = (dev(rng.standard_normal((B, NH, S, dqk)), BF) for _ in range(2))
    v = dev(rng.standard_normal((B, NH, S, dv)), BF)
    i, f = (dev(a, BF) for a in gates(rng, (B, NH, S)))
    f[:, 1::2] -= 5
    st = tuple(dev(rng.standard_normal(s) * 0.1) for s in ((B, NH, dqk, dv), (B, NH, dqk), (B, NH)))
    try:
        ops.chunkwise_segments(P)
        for _ in range(3):
            h, s1 = ops.mlstm_chunkwise(q, k, v, i, f, st)
            for hd in (0, 1, NH - 1):
                one = slice(hd, hd + 1)
                ho, so = ops.mlstm_chunkwise(*(a[-1:, one] for a in (q, k, v, i, f)), tuple(s[-1:, one].contiguous() for s in st))
                assert torch.equal(h[-1:, one], ho)
                for a, b in zip(s1, so):
                    assert torch.equal(a[-1:, one], b)
    finally:
        ops.chunkwise_segments(None)


@pytest.mark.parametrize("S", [128, 4096, 4224])
def test_chunkwise_gate_prepass_forms_and_mixed_heads(ops, S):
    """1, 32 and 33 tiles: the one-launch gate pre-pass, its last size, and the three-launch form; one head of bounded gate
    spread beside one that forgets within a token, so both tensor-core paths share the launches; one pass and segments."""
    rng = np.random.default_rng(S)
    NH, d = 2, 128
    q, k, v = (xo.bf16_round(rng.standard_normal((1, NH, S, d)).astype(np.float32)) for _ in range(3))
    i, f = (a.astype(np.float32) for a in gates(rng, (1, NH, S)))
    f[:, 1] -= 8
    i, f = xo.bf16_round(i), xo.bf16_round(f)
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f)
    args = [dev(a, torch.bfloat16) for a in (q, k, v, i, f)]
    try:
        for P in (1, 3):
            ops.chunkwise_segments(P)
            h, st = ops.mlstm_chunkwise(*args)
            assert relerr(host(h), h_ref) < BF16_TOL
            for a, r in zip(st, st_ref):
                assert relerr(host(a), r) < BF16_TOL
    finally:
        ops.chunkwise_segments(None)


@pytest.mark.parametrize("general", [False, True])
def test_chunkwise_segment_parallel_equals_single_pass(ops, general):
    """The segment-parallel two-pass mode (every segment from an empty state, states combined, every segment again
    from its true start state) against the single pass and against the oracle: bf16 tensor-core shapes, with a
    carried-in state and a sequence tail, for segment counts that divide the tiles evenly and unevenly."""
    rng = np.random.default_rng(21)
    B, NH, S, dqk, dv = 1, 2, 2048 + 70, 256, 256
    q, k = (xo.bf16_round(rng.standard_normal((B, NH, S, dqk)).astype(np.float32)) for _ in range(2))
    v = xo.bf16_round(rng.standard_normal((B, NH, S, dv)).astype(np.float32))
    i, f = (xo.bf16_round(a) for a in gates(rng, (B, NH, S)))
    st0 = ((rng.standard_normal((B, NH, dqk, dv)) * 0.1).astype(np.float32),
           (rng.standard_normal((B, NH, dqk)) * 0.1).astype(np.float32), rng.standard_normal((B, NH)).astype(np.float32))
    h_ref, st_ref = xo.mlstm_recurrent(q, k, v, i, f, st0)
    args = [dev(a, torch.bfloat16) for a in (q, k, v, i, f)]
    std = tuple(dev(a) for a in st0)
    try:
        ops.chunkwise_general_only(general)
        ops.chunkwise_segments(1)
        h1, s1 = ops.mlstm_chunkwise(*args, state=std)
        for P in (2, 3, 4, 16):
            ops.chunkwise_segments(P)
            h, s = ops.mlstm_chunkwise(*args, state=std)
            assert relerr(host(h), h_ref) < BF16_TOL and relerr(host(h), host(h1)) < BF16_TOL, P
            assert relerr(host(s[0]), st_ref[0]) < BF16_TOL and relerr(host(s[1]), st_ref[1]) < BF16_TOL, P
            assert np.abs(host(s[2]) - st_ref[2]).max() < 1e-3, P
            assert relerr(host(s[0]), host(s1[0])) < 5e-3, P
        ops.chunkwise_segments(None)     # planned from the grid size: 4 CTAs on 148 SMs -> segments
        h, s = ops.mlstm_chunkwise(*args, state=std)
        assert relerr(host(h), h_ref) < BF16_TOL and relerr(host(s[0]), st_ref[0]) < BF16_TOL
    finally:
        ops.chunkwise_segments(None)
        ops.chunkwise_general_only(False)


def test_bounded_wait_gives_up_and_status_queries_report_ok(ops):
    """Device-side time-outs without hanging anything: (a) the bounded mbarrier wait of the tensor-core kernels,
    built with a tiny poll limit in a test-only kernel, on a barrier nobody arrives at - it must return false,
    raise the abort flag (which releases every other role) and let the kernel end normally; (b) after real
    forwards the status queries of the C ABI report no time-out."""
    import ctypes
    sys_path = Path(__file__).resolve().parent / "helpers"
    sys.path.insert(0, str(sys_path))
    from build_helpers import build
    lib = ctypes.CDLL(str(build()))
    out = (ctypes.c_int * 3)()
    assert lib.timeout_probe_run(out) == 0
    assert list(out) == [0, 0, 1]
    rng = np.random.default_rng(2)
    B, NH, S, dqk, dv = 1, 1, 256, 128, 128
    q, k = (dev(rng.standard_normal((B, NH, S, dqk)).astype(np.float32), torch.bfloat16) for _ in range(2))
    v = dev(rng.standard_normal((B, NH, S, dv)).astype(np.float32), torch.bfloat16)
    i, f = (dev(a, torch.bfloat16) for a in gates(rng, (B, NH, S)))
    ws = torch.empty(ops.chunkwise_workspace_bytes(B, NH, S, dqk, dv, 64, torch.bfloat16), dtype=torch.uint8, device="cuda")
    ops.mlstm_chunkwise(q, k, v, i, f, workspace=ws)
    ops.chunkwise_status(ws)            # raises on XLSTM_ERR_TIMEOUT
    ops.slstm_recurrent_status()


@pytest.mark.parametrize("dtype,S,full", [(torch.float32, 200, True), (torch.float32, 40, True), (torch.float32, 200, False),
                                          (torch.bfloat16, 200, True)])
def test_status_after_forwards_without_waits(ops, dtype, S, full):
    """The fp32 kernels (fp32 inputs, and bf16 head shapes outside the tensor-core kernels) cannot time out: whatever the
    scratch held before, and with a stabiliser that is not zero, the status of a forward that was handed it is fine; with scratch
    too small for the chunk states too."""
    rng = np.random.default_rng(S)
    B, NH, d = 1, 2, 64
    q, k, v = (dev(rng.standard_normal((B, NH, S, d)).astype(np.float32), dtype) for _ in range(3))
    i, f = (dev(a, dtype) for a in gates(rng, (B, NH, S)))
    st = tuple(dev(a) for a in (rng.standard_normal((B, NH, d, d)).astype(np.float32),
                                rng.standard_normal((B, NH, d)).astype(np.float32), np.full((B, NH), 2.5, np.float32)))
    need = max(ops.chunkwise_workspace_bytes(B, NH, S, d, d, 64, dtype), 256)
    ws = torch.full((need if full else 256,), 255, dtype=torch.uint8, device="cuda")
    h, st1 = ops.mlstm_chunkwise(q, k, v, i, f, state=st, workspace=torch.full_like(ws, 255))
    from xlstm_cuda import _lib
    code = _lib.F32 if dtype == torch.float32 else _lib.BF16
    h2, C, n, m = torch.empty_like(h), *(torch.empty_like(a) for a in st1)
    rc = _lib.load().xlstm_mlstm_chunkwise_fwd(*(a.data_ptr() for a in (q, k, v, i, f, *st, h2, C, n, m)), B, NH, S, d, d, 64, 1e-6,
                                               code, None, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    ops.chunkwise_status(ws)
    assert relerr(host(h2), host(h)) < FP32_TOL and relerr(host(C), host(st1[0])) < FP32_TOL


def test_chunkwise_scatter_entry_point_single_rank(ops):
    """The token-sharded store mode with one rank: h lands in the [B, S, NH, dv] buffer exactly as the regular
    entry point writes it into a strided view of the same layout (the multi-rank routing is covered by the
    two-GPU test)."""
    from xlstm_cuda.parallel import FusedHeadScatter
    rng = np.random.default_rng(31)
    B, NH, S, dqk, dv = 2, 2, 512, 128, 256
    q, k = (dev(rng.standard_normal((B, NH, S, dqk)).astype(np.float32), torch.bfloat16) for _ in range(2))
    v = dev(rng.standard_normal((B, NH, S, dv)).astype(np.float32), torch.bfloat16)
    i, f = (dev(a, torch.bfloat16) for a in gates(rng, (B, NH, S)))
    w = dev((rng.standard_normal((NH * dv, 48)) * 0.05).astype(np.float32), torch.bfloat16)
    h, st = ops.mlstm_chunkwise(q, k, v, i, f)
    sc = FusedHeadScatter(B, S, NH, dv, torch.bfloat16, "cuda")
    y, st2 = sc.run(q, k, v, i, f, None, out_proj=w)
    assert torch.equal(sc.buf, h.permute(0, 2, 1, 3).contiguous())
    assert all(torch.equal(a, b) for a, b in zip(st, st2))
    assert torch.equal(y, h.permute(0, 2, 1, 3).reshape(B, S, NH * dv) @ w)
