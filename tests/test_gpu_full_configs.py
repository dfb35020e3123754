"""GPU parity at the FULL shapes of the benchmark configurations (bf16, fp32 state, tolerance 2e-2 =
max|a-b| / max|b|), against fixtures made by running the reference's own classes on CPU
(tests/golden/make_golden_full.py) and against the CPU oracle where it finishes in seconds."""
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

from conftest import relerr
from oracle import oracle as xo

sys.path.insert(0, str(Path(__file__).resolve().parent / "golden"))
from make_golden_full import block_7b_input, extreme_inputs, recurrent_fp64  # noqa: E402
from param_init import fill_parameters  # noqa: E402

pytestmark = pytest.mark.gpu
BF16_TOL = 2e-2
bf = torch.bfloat16


def host(t):
    return t.detach().float().cpu().numpy()


def from_bits(a):
    return torch.from_numpy(a.view(np.int16).copy()).view(torch.bfloat16).float().numpy()


@pytest.mark.parametrize("fused", [True, False])
def test_mlstm_block_7b_shape_bf16_teacher_forced(golden, fused):
    """The 7B-shaped model, one layer: the reference mLSTMBlock at D=4096, NH=8 (256/512, FFN 10944) with bf16
    parameters (N(0, 0.02) matrices) and compute and fp32 state.  192 tokens (one 128-token tile on the tensor
    cores + a 64-token tail) in one call, then 8 single-token calls through the decode path, all on the
    reference's own input.  The fixture holds the reference's bf16 run AND its fp32 evaluation of the same
    rounded parameters: a chain of bf16 GEMMs, norms and the cell is not reproducible to 2e-2 between two bf16
    implementations (the reference's own bf16 run is 1.4-2.2e-2 away from its fp32 run here), so every
    quantity is held to 2e-2 against the fp32 evaluation and to 2e-2 plus the reference's own distance against
    its bf16 run.  Follows xlstm_metal/torch_native/blocks/mlstm/mlstm_block.py:192-206, mlstm_neuron.py:142-162."""
    from make_golden_full import fill_block_7b
    from xlstm_cuda.blocks import mLSTMBlock
    g = golden("block_7b_bf16")
    blk = mLSTMBlock(0, embedding_dim=4096, num_heads=8, compute_dtype=bf, state_dtype=torch.float32).eval()
    fill_block_7b(blk, int(g["seed_params"]))
    blk = blk.to(bf).cuda()
    if fused:
        blk.fuse_projections()
    x = block_7b_input(int(g["seed_input"])).cuda()
    P = int(g["prefill_tokens"])

    def check(name, got, ref16, ref32):
        own = relerr(ref16, ref32)
        e32, e16 = relerr(got, ref32), relerr(got, ref16)
        assert e32 < BF16_TOL and e16 < BF16_TOL + own, (name, e32, e16, own)

    def check_m(got, ref16, ref32):   # the stabiliser: absolute; the reference's bf16 log-sigmoid makes its own m noisy
        own = np.abs(ref16 - ref32).max()
        assert np.abs(got - ref32).max() < BF16_TOL and np.abs(got - ref16).max() < BF16_TOL + own

    y16, y32 = from_bits(g["y_cols"]), from_bits(g["y32_cols"])
    with torch.inference_mode():
        y_pre, st = blk(x[:, :P], None)
        branch, _ = blk.mlstm_cell(blk.norm_mlstm(x[:, :P]), None)
        check("mlstm branch", host(branch)[:, :, ::8], from_bits(g["mlstm_cols"]), from_bits(g["mlstm32_cols"]))
        check("y", host(y_pre)[:, :, ::8], y16[:, :P], y32[:, :P])
        C, n, m = st
        assert C.dtype == torch.float32 and C.shape == (1, 8, 256, 512)
        check("C", host(C)[:, :, ::8, ::8], g["C_pre"], g["C32_pre"])
        check("n", host(n), g["n_pre"], g["n32_pre"])
        check_m(host(m), g["m_pre"], g["m32_pre"])
        ys = []
        for t in range(P, x.shape[1]):
            if fused:
                assert blk._token_step_ok(x[:, t:t + 1])
            yt, st = blk(x[:, t:t + 1], st)
            ys.append(yt)
        check("y steps", host(torch.cat(ys, 1))[:, :, ::8], y16[:, P:], y32[:, P:])
        C, n, m = st
        check("C end", host(C)[:, :, ::8, ::8], g["C_end"], g["C32_end"])
        check("n end", host(n), g["n_end"], g["n32_end"])
        check_m(host(m), g["m_end"], g["m32_end"])


def test_slstm_block_diagonal_config4_shape_bf16(golden):
    """The sLSTM stack, one block: d=1024, 4 heads x 256, bf16, B=4, S=64 - the tensor-core recurrence,
    the padded FFN and the fused LayerNorm together.  The reference class
    (kernel_development/xlstm/implementations/pytorch/xlstm_pytorch_enhanced.py:367-488) does not run with bf16
    parameters, so the fixture is its fp32 run on the bf16-rounded parameters and input."""
    from xlstm_cuda.blocks import sLSTMBlockDiag
    g = golden("slstm_blockdiag_bf16_1024")

    class Cfg:
        inp_dim, head_dim, head_num, p_factor, norm_eps, gate_soft_cap = 1024, 256, 4, (2.0, 4 / 3), 1e-6, 15.0
    blk = sLSTMBlockDiag(Cfg()).eval()
    named = dict(blk.named_parameters())
    fill_parameters(named, seed=int(g["seed_params"]))
    with torch.no_grad():
        for name, prm in named.items():
            if ".R_" in name or name.startswith("R_"):
                prm.mul_(0.02 / 0.3)
    blk = blk.to(bf).cuda()
    x = torch.from_numpy(np.random.default_rng(int(g["seed_input"])).standard_normal((4, 64, 1024)).astype(np.float32)).to(bf).cuda()
    with torch.inference_mode():
        y, st = blk(x)
    assert relerr(host(y)[:, :, ::2], g["y_fp32_of_bf16_params"]) < BF16_TOL
    for got, key in zip(st, "cnhm"):
        assert got.dtype == torch.float32
        assert relerr(host(got), g[key]) < BF16_TOL, key


def test_chunkwise_config3_full_length_final_state_and_last_tokens():
    """Full length: S = 32768 at 256/512, bf16.  The last 256 tokens of h and the final (C, n, m)
    against the CPU oracle's step-by-step recurrence over all 32768 tokens (follows
    xlstm_metal/torch_native/blocks/mlstm/mlstm_chunkwise/mlstm_recurrent_kernel_cell.py:106-153), through both
    tensor-core kernels."""
    from xlstm_cuda import ops
    B, NH, S, dqk, dv = 1, 4, 32768, 256, 512
    g = torch.Generator().manual_seed(33)
    q = torch.randn(B, NH, S, dqk, generator=g).to(bf)
    k = torch.randn(B, NH, S, dqk, generator=g).to(bf)
    v = torch.randn(B, NH, S, dv, generator=g).to(bf)
    i = (15 * torch.tanh(torch.randn(B, NH, S, generator=g) / 15)).to(bf)
    f = (15 * torch.tanh((torch.randn(B, NH, S, generator=g) + 3) / 15)).to(bf)
    h_ref, st_ref = xo.mlstm_recurrent(*(t.float().numpy() for t in (q, k, v, i, f)))
    args = [t.cuda() for t in (q, k, v, i, f)]
    try:
        for general in (False, True):
            ops.chunkwise_general_only(general)
            h, st = ops.mlstm_chunkwise(*args)
            assert torch.isfinite(h.float()).all()
            assert relerr(host(h[:, :, -256:]), h_ref[:, :, -256:]) < BF16_TOL, general
            assert relerr(host(h[:, :, 16000:16256]), h_ref[:, :, 16000:16256]) < BF16_TOL, general
            assert relerr(host(st[0]), st_ref[0]) < BF16_TOL and relerr(host(st[1]), st_ref[1]) < BF16_TOL, general
            assert np.abs(host(st[2]) - st_ref[2]).max() < 1e-3, general
    finally:
        ops.chunkwise_general_only(False)


def test_chunkwise_extreme_gates_no_worse_than_the_reference_bf16_cell(golden):
    """Gates pinned at the soft-cap limits: on the tokens where the normaliser nearly cancels (|h| > 5 in float64)
    ANY bf16 evaluation is far from float64.  The fixture holds the per-token error of the reference's own cell
    run with compute_dtype=bfloat16 on these inputs; the kernel must not be worse than it there, and must meet
    the bf16 tolerance everywhere else."""
    from xlstm_cuda import ops
    g = golden("mlstm_extreme_bf16")
    q, k, v, i, f = extreme_inputs()
    h64, st64 = recurrent_fp64(q, k, v, i, f)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", bf)
    h, st = ops.mlstm_chunkwise(*(dev(a) for a in (q, k, v, i, f)))
    assert np.isfinite(host(h)).all()
    err = np.abs(host(h) - h64).max(-1)
    mag = g["h64_mag_tok"]
    big = mag > 5.0
    assert 0.2 < big.mean() < 0.6
    ours, ref = err[big] / mag[big], g["ref_err_tok"][big] / mag[big]
    assert np.median(ours) <= np.median(ref) and np.quantile(ours, 0.95) <= np.quantile(ref, 0.95)
    assert relerr(np.where(big[..., None], 0.0, host(h)), np.where(big[..., None], 0.0, h64)) < BF16_TOL
    assert relerr(host(st[0]), st64[0]) < BF16_TOL
