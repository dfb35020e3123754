"""The work this framework is used for, as a list of cases that can be timed and compared.

Two levels are listed, because users enter at both: the recurrent cells with their drop-in signature
``cell(q, k, v, i, f, state) -> (h, state)``, and the blocks / models above them (``xLSTMRunner``, ``WiredxLSTM``,
``sLSTMBlockDiag``, ``sLSTMBlock``).  The path is an inference path: its directions are prefill (many tokens) and
decode (one token per sequence), both with and without a carried state.

Head shapes are the ones the configurations, tests and benchmark of this repository use: 256/512 (the 7B-shaped
model), 128/256, 64/128 and 64/64.
"""
import math
import sys
import tempfile
from pathlib import Path

import torch

# the package folder has a dash in its parent's name, so it is reached through the path (as the tests do); the
# working folder is the repository's root
_PKG = str(Path.cwd() / "xlstm-metal_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from xlstm_cuda.blocks import mLSTMParallelKernelCell, mLSTMRecurrentKernelCell, sLSTMBlock, sLSTMBlockDiag  # noqa: E402
from xlstm_cuda.generate import xLSTMRunner  # noqa: E402
from xlstm_cuda.utils import XLSTM_7B_CONFIG, write_model_dir  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
CHUNK = 64           # chunk size of every configuration
GATE_CAP = 15.0


def listed():
    return [
        # one decode step of one sequence: the smallest call a generation loop makes into the cell
        _step("step_b1_bf16", B=1, NH=8, dqk=256, dv=512, dtype="bf16"),
        # one decode step of a serving batch at the 7B head shape: the framework's headline workload
        _step("step_b16_bf16", B=16, NH=8, dqk=256, dv=512, dtype="bf16"),
        # long-sequence prefill at the 7B head shape: the largest cell call
        _prefill("prefill_b4_s32768_bf16", B=4, NH=8, S=32768, dqk=256, dv=512, dtype="bf16", gates="usual", state=False),
        # the next part of a prompt that is fed in parts: ordinary length, state carried in
        _prefill("prefill_b1_s2048_bf16_carried", B=1, NH=8, S=2048, dqk=256, dv=512, dtype="bf16", gates="usual", state=True),
        # two ragged prompts whose heads have different time scales (half of them forget within a few tokens)
        _prefill("prefill_b2_s4001_bf16_mixed", B=2, NH=8, S=4001, dqk=256, dv=512, dtype="bf16", gates="mixed", state=False),
        # a small layer in the package's default dtype, fp32: short prompt, few narrow heads
        _prefill("prefill_b1_s256_fp32", B=1, NH=4, S=256, dqk=64, dv=64, dtype="fp32", gates="usual", state=False),
        # fp32 at the 7B head shape
        _prefill("prefill_b2_s1024_fp32", B=2, NH=8, S=1024, dqk=256, dv=512, dtype="fp32", gates="usual", state=False),
        # a prompt of 31 chunks (no whole number of the kernel's 128-token tiles) through half the depth of the 7B-shaped
        # model (its blocks are all alike): logits of every position
        _model("model_prompt_s1984", B=1, S=1984, blocks=16, graph=False),
        # one token of one sequence through the same, captured as a CUDA graph like every decode loop
        _model("model_token_b1_graph", B=1, S=1, blocks=16, graph=True),
        # one token of 16 sequences through a quarter of that model, called as it is (no graph)
        _model("model_token_b16", B=16, S=1, blocks=8, graph=False),
        # a stack of sLSTM blocks with block-diagonal recurrent weights over a training-length batch
        _sdiag("slstm_stack_b32_s1024", B=32, S=1024, heads=4, dh=256, blocks=4, dtype="bf16"),
        # an sLSTM block as the model wiring builds it (scalar gates per head, causal conv, SwiGLU FFN)
        _sblock("slstm_block_b4_s2048", B=4, S=2048, d=4096, heads=4, dtype="bf16"),
    ]


def draw(rng):
    kind = rng.choice(["step", "prefill_bf16", "prefill_bf16", "prefill_fp32", "prompt", "token", "sdiag", "sblock"])
    heads = [(256, 512), (256, 512), (128, 256), (64, 128), (64, 64)]
    if kind == "step":
        dqk, dv = rng.choice(heads)
        return _step(None, B=_log(rng, 1, 64), NH=rng.choice([2, 4, 8]), dqk=dqk, dv=dv,
                     dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "prefill_bf16":
        dqk, dv = rng.choice(heads)
        B = _log(rng, 1, 8)
        return _prefill(None, B=B, NH=rng.choice([1, 2, 4, 8]), S=_log(rng, 128, 4 * 32768 // B if B > 4 else 32768),
                        dqk=dqk, dv=dv, dtype="bf16", gates=rng.choice(["usual", "usual", "mixed"]), state=rng.random() < 0.5)
    if kind == "prefill_fp32":
        dqk, dv = rng.choice(heads)
        B = _log(rng, 1, 4)
        return _prefill(None, B=B, NH=rng.choice([2, 4, 8]), S=_log(rng, 2, 4096 // B), dqk=dqk, dv=dv, dtype="fp32",
                        gates=rng.choice(["usual", "usual", "mixed"]), state=rng.random() < 0.5)
    if kind == "prompt":
        # whole chunks of 64 tokens, an odd number of them as likely as an even one
        return _model(None, B=rng.choice([1, 1, 2]), S=CHUNK * _log(rng, 2, 32), blocks=rng.randint(1, 6), graph=False)
    if kind == "token":
        return _model(None, B=_log(rng, 1, 64), S=1, blocks=rng.randint(1, 6), graph=rng.random() < 0.5)
    if kind == "sdiag":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        return _sdiag(None, B=_log(rng, 1, 32), S=_log(rng, 1, 1024), heads=rng.choice([2, 4]), dh=rng.choice([64, 128, 256]),
                      blocks=1 if dtype == "fp32" else rng.randint(1, 3), dtype=dtype)
    return _sblock(None, B=_log(rng, 1, 8), S=_log(rng, 1, 4096), d=rng.choice([1024, 2048, 4096]), heads=4,
                   dtype=rng.choice(["bf16", "bf16", "fp32"]))


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm (odd ones as likely as even ones)."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _case(name, kind, **kw):
    case = {"kind": kind, **kw}
    if name:
        case["name"] = name
    return case


def _step(name, **kw):
    return _case(name, "step", **kw)


def _prefill(name, **kw):
    return _case(name, "prefill", **kw)


def _model(name, **kw):
    return _case(name, "model", **kw)


def _sdiag(name, **kw):
    return _case(name, "sdiag", **kw)


def _sblock(name, **kw):
    return _case(name, "sblock", **kw)


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape, mean=0.0, std=1.0):
    return torch.randn(*shape, generator=gen, device="cuda") * std + mean


def _cap(x):
    return GATE_CAP * torch.tanh(x / GATE_CAP)


def _mlstm_inputs(case, gen):
    """q, k, v ~ N(0,1) and gates in the layout the projections leave them in: [B,S,NH,d] seen as [B,NH,S,d].
    ``usual`` gates: i ~ N(0,1), f ~ N(3,1) (a head remembers some twenty tokens); ``mixed``: every second head has
    f ~ N(-2,1) and forgets within a token or two.  Carried state: C, n ~ N(0,0.1), m = 0."""
    B, NH, S, dqk, dv, dt = case["B"], case["NH"], case.get("S", 1), case["dqk"], case["dv"], DTYPES[case["dtype"]]
    heads = lambda d: _randn(gen, B, S, NH, d).to(dt).permute(0, 2, 1, 3)
    q, k, v = heads(dqk), heads(dqk), heads(dv)
    i = _cap(_randn(gen, B, S, NH)).to(dt).permute(0, 2, 1)
    f = _randn(gen, B, S, NH, mean=3.0)
    if case.get("gates") == "mixed":
        f[..., 1::2] -= 5.0
    f = _cap(f).to(dt).permute(0, 2, 1)
    state = None
    if case.get("state", True):
        state = (_randn(gen, B, NH, dqk, dv, std=0.1), _randn(gen, B, NH, dqk, std=0.1), torch.zeros(B, NH, device="cuda"))
    return q, k, v, i, f, state


def _init_model(module, gen, fgate_bias):
    """Weights ~ N(0,0.02), norm weights 1, biases 0, forget-gate biases spread over [3, 6].  As in trained models the
    residual stream is not swamped by any one block: embeddings ~ N(0,1), and the projections that write into the
    stream are scaled by the usual 1 / sqrt(2 x depth), taken at the depth of the full model."""
    into_stream = ("out_proj.weight", "ffn_proj_down.weight", "down_proj.weight")
    with torch.no_grad():
        for name, prm in module.named_parameters():
            if prm.dim() >= 2:
                prm.normal_(0.0, 1.0 if name.endswith("embedding.weight") else 0.02, generator=gen)
                if name.endswith(into_stream):
                    prm.mul_((2 * XLSTM_7B_CONFIG["num_blocks"]) ** -0.5)
            elif name.endswith(fgate_bias):
                prm.copy_(torch.linspace(3.0, 6.0, prm.numel()))
            elif name.endswith("bias"):
                prm.zero_()


class _DiagConfig:
    """Configuration of ``sLSTMBlockDiag`` at the benchmark's proportions (FFN factor 4/3)."""

    def __init__(self, heads, dh):
        self.inp_dim, self.head_dim, self.head_num = heads * dh, dh, heads
        self.p_factor, self.norm_eps, self.gate_soft_cap = (2.0, 4 / 3), 1e-6, GATE_CAP


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "step":
        cell = mLSTMRecurrentKernelCell(case["NH"], case["dqk"], case["dv"], compute_dtype=DTYPES[case["dtype"]])
        return {"case": case, "cell": cell, "args": _mlstm_inputs(case, gen)}
    if kind == "prefill":
        cell = mLSTMParallelKernelCell(case["NH"], case["dqk"], case["dv"], CHUNK, compute_dtype=DTYPES[case["dtype"]])
        return {"case": case, "cell": cell, "args": _mlstm_inputs(case, gen)}
    if kind == "model":
        return _prepare_model(case, gen)
    if kind == "sdiag":
        D, dt = case["heads"] * case["dh"], DTYPES[case["dtype"]]
        blocks = []
        with torch.device("cuda"):
            for _ in range(case["blocks"]):
                blk = sLSTMBlockDiag(_DiagConfig(case["heads"], case["dh"]))
                _init_model(blk, gen, "W_f.bias")
                blocks.append(blk.to(dt))
        return {"case": case, "blocks": blocks, "x": _randn(gen, case["B"], case["S"], D).to(dt)}
    dt = DTYPES[case["dtype"]]
    with torch.device("cuda"):
        blk = sLSTMBlock(0, embedding_dim=case["d"], num_heads=case["heads"])
    _init_model(blk, gen, "fgate_proj.bias")
    return {"case": case, "block": blk.to(dt).eval(), "x": _randn(gen, case["B"], case["S"], case["d"]).to(dt)}


def _prepare_model(case, gen):
    with tempfile.TemporaryDirectory() as tmp:
        path = write_model_dir(tmp, dict(XLSTM_7B_CONFIG, num_blocks=case["blocks"]))
        runner = xLSTMRunner(str(path), device=torch.device("cuda"))
    _init_model(runner.model, gen, "fgate_proj.bias")
    B, S = case["B"], case["S"]
    ids = torch.randint(0, XLSTM_7B_CONFIG["vocab_size"], (B, S), generator=gen, device="cuda")
    st = {"case": case, "runner": runner, "ids": ids, "state": None}
    if S == 1:   # a decode step continues a sequence: the states a prompt of 128 tokens leaves
        with torch.inference_mode():
            prompt = torch.randint(0, XLSTM_7B_CONFIG["vocab_size"], (B, 128), generator=gen, device="cuda")
            runner.forward(prompt)
        st["state"] = runner.state
    if case["graph"]:
        def token():
            return runner.model(ids, st["state"], return_last_states=True)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side), torch.inference_mode():
            token()
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.inference_mode(), torch.cuda.graph(st["graph"]):
            st["out"] = token()
    return st


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("step", "prefill"):
        q, k, v, i, f, state = st["args"]
        with torch.inference_mode():
            h, (C, n, m) = st["cell"](q, k, v, i, f, state)
        return {"h": h, "C": C, "n": n, "m": m}
    if kind == "model":
        if case["graph"]:
            st["graph"].replay()
            logits, states = st["out"]
        else:
            runner = st["runner"]
            runner.state = st["state"]
            logits, states = runner.forward(st["ids"]), runner.state
        return {"logits": logits, "C": [s[0] for s in states], "n": [s[1] for s in states], "m": [s[2] for s in states]}
    if kind == "sdiag":
        y, states = st["x"], []
        with torch.inference_mode():
            for blk in st["blocks"]:
                y, s = blk(y)
                states.append(s)
        return {"y": y, "states": states}
    with torch.inference_mode():
        y, state = st["block"](st["x"], None)
    return {"y": y, "state": state}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _cell_work(B, NH, S, dqk, dv, esz, state_in):
    """Chunkwise recurrence: state update and read-out (4 dqk dv per token) and, for several tokens, the causal half
    of the in-chunk products (L (dqk + dv)); inputs and outputs once, the fp32 state out and, if carried, in."""
    L = min(S, CHUNK)
    flops = B * NH * S * (4 * dqk * dv + (L * (dqk + dv) if S > 1 else dqk * dv))
    state = B * NH * (dqk * dv + dqk + 1) * 4
    return B * NH * S * (2 * dqk + 2 * dv + 2) * esz + state * (2 if state_in else 1), flops


def work(case):
    kind = case["kind"]
    if kind in ("step", "prefill"):
        b, f = _cell_work(case["B"], case["NH"], case.get("S", 1), case["dqk"], case["dv"], 2 if case["dtype"] == "bf16" else 4,
                          case.get("state", True))
        return {"bytes": b, "flops": f}
    B, S = case["B"], case["S"]
    tokens = B * S
    if kind == "model":
        d, vocab, NH = XLSTM_7B_CONFIG["embedding_dim"], XLSTM_7B_CONFIG["vocab_size"], XLSTM_7B_CONFIG["num_heads"]
        ffn = -(-int(d * XLSTM_7B_CONFIG["ffn_proj_factor"]) // 64) * 64
        linear = case["blocks"] * (d * (d + d + d + d + 2 * NH) + 3 * d * ffn) + vocab * d   # q,k: d/2 each; v, o, out; i, f
        _, cell_f = _cell_work(B, NH, S, d // 2 // NH, d // NH, 2, S == 1)
        state = B * NH * (d // 2 // NH) * (d // NH) * 4 * (2 if S == 1 else 1) * case["blocks"]
        return {"bytes": linear * 2 + state + tokens * (8 + d * 2 + vocab * 2),
                "flops": 2 * linear * tokens + case["blocks"] * cell_f}
    esz = 2 if case["dtype"] == "bf16" else 4
    if kind == "sdiag":
        D = case["heads"] * case["dh"]
        proj = int(4 / 3 * D)
        weights = 4 * D * D + 4 * D * case["dh"] + 3 * D * proj
        return {"bytes": case["blocks"] * (weights * esz + 4 * B * D * 4) + 2 * tokens * D * esz,
                "flops": case["blocks"] * 2 * weights * tokens}
    d = case["d"]
    ffn = -(-int(d * 2.667) // 64) * 64
    weights = 2 * d * d + 3 * d * ffn + 3 * d * case["heads"] + 4 * d
    return {"bytes": weights * esz + 2 * tokens * d * esz + B * (2 * d + case["heads"]) * 4, "flops": 2 * weights * tokens}


def tolerance(case):
    """About four times the distance measured on a B200 to another correct evaluation: the cells against the exact fp32
    recurrence on the same inputs (bf16: h 2.9e-3 from the bf16 operands of the in-chunk products, 1.7e-3 from the
    rounding of h alone; C 1.7e-3) or against float64 (fp32: h 1.1e-6, the weakly normalised rows dominate), the models
    against themselves with the projections as separate GEMMs and the other prefill kernel (C of the last block 3.4e-2
    at 16 blocks, 1.6e-2 at 5, 1.2e-3 at 2)."""
    kind, fp32 = case["kind"], case.get("dtype", "bf16") == "fp32"
    if kind == "model":
        return {"rel": 0.02 * math.sqrt(case["blocks"])}
    if kind == "sdiag":
        # the stabiliser m grows by up to the forget-gate bias a step, so the exponents lose bits with S even in fp32
        # (c, n 2.7e-4 from float64 after 1024 steps)
        return {"rel": 1e-5 + 1e-6 * case["S"] if fp32 else 3e-2}
    if kind == "sblock":
        return {"rel": 5e-6 if fp32 else 3e-2}      # fp32 1.2e-6 from float64, bf16 8.3e-3 from fp32
    if fp32:
        return {"rel": 5e-6}
    return {"rel": 7e-3 if kind == "step" else 1.2e-2}
