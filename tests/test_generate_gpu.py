"""Decoding with a KV cache (extension) against the oracle's full-sequence model, on a B200.

The reference has no decoder (README.md:148 lists it as a later milestone); its model is
scripts/gpt2_torch.py's, so the logits the decoder leaves after a position must be the
model's logits at that position of the whole sequence. The oracle runs the FP32 model with
the weights the decoder computes with (matrices rounded to FP16, or their per-row int8
approximation), so the bound is the kernels' own error: relative L2 <= 5e-3 on a position's
logits (FP16 activations under FP32 accumulation, as for the training forward pass).
"""

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

import flint_b200
import flint_oracle as oracle
from flint_b200.generate import Generator

pytestmark = pytest.mark.gpu
DEV = "cuda"
SMALL = dict(n_layer=2, n_head=2, n_embd=128, block_size=64, vocab_size=200, padded_vocab_size=208)


def u16(t):
    return torch.from_numpy(t.numpy().astype(np.uint16).view(np.int16)).to(DEV)


def rel_l2(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-300)).item()


def weights(cfg, seed=1234):
    params = oracle.gpt2_init(cfg, seed=seed)
    g = torch.Generator().manual_seed(seed + 1)
    for name, p in params.items():                      # nothing trivially 0 or 1
        if name.endswith(".bias") and "ln_" not in name:
            params[name] = torch.randn(p.shape, generator=g) * 0.02
        elif "ln_" in name:
            params[name] = p + torch.randn(p.shape, generator=g) * 0.05
    return params


def model_for(flint, cfg, params):
    config = flint_b200.Gpt2Config(cfg["n_layer"], cfg["n_head"], cfg["n_embd"], cfg["block_size"],
                                   cfg["vocab_size"], cfg["padded_vocab_size"], 1, 8, 0, 0)
    model = flint_b200.Gpt2(flint, config, True)
    model.load({k: v.to(DEV) for k, v in params.items()})
    return model


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
@pytest.mark.parametrize("sequences", [3, 12])
def test_prefill_and_teacher_forced_steps_match_the_full_model(flint, sequences, int8):
    """A prompt of 16 tokens, then 12 given tokens one at a time: the logits after each
    position against the oracle's logits of the whole 28-token sequence."""
    params = weights(SMALL)
    prompt, steps = 16, 12
    g = torch.Generator().manual_seed(3)
    tokens = torch.randint(0, SMALL["vocab_size"], (sequences, prompt + steps), generator=g)
    want = oracle.gpt2_decode_logits(SMALL, params, tokens, int8=int8)
    model = model_for(flint, SMALL, params)
    try:
        with Generator(flint, model, sequences, 64, int8) as gen:
            gen.prefill(u16(tokens[:, :prompt]))
            assert gen.position() == prompt
            assert rel_l2(gen.logits().cpu(), want[:, prompt - 1]) <= 5e-3
            for t in range(prompt, prompt + steps):
                chosen = gen.step(u16(tokens[:, t])).cpu().to(torch.int64) & 0xFFFF
                got = gen.logits().cpu()
                assert rel_l2(got, want[:, t]) <= 5e-3, t
                assert torch.equal(chosen, got.argmax(1)), t          # greedy = argmax of its logits
                assert int(chosen.max()) < SMALL["vocab_size"]
            assert gen.position() == prompt + steps
    finally:
        model.close()
    assert not flint.kernel_fault()


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
@pytest.mark.parametrize("layers, sequences, heads, prompt", [(1, 1, 2, 8), (1, 20, 4, 24), (3, 64, 2, 8), (2, 5, 14, 136)])
def test_prompt_logits_come_from_the_last_rows_alone(flint, layers, sequences, heads, prompt, int8):
    """Behind the last block's attention a prompt goes on with one row per sequence, on the decode
    kernels: 1 to 64 rows, a model whose first block is its last, and the cache that a step then reads."""
    cfg = dict(n_layer=layers, n_head=heads, n_embd=64 * heads, block_size=160, vocab_size=200, padded_vocab_size=208)
    params = weights(cfg)
    g = torch.Generator().manual_seed(7)
    tokens = torch.randint(0, 200, (sequences, prompt + 1), generator=g)
    want = oracle.gpt2_decode_logits(cfg, params, tokens, int8=int8)
    model = model_for(flint, cfg, params)
    try:
        with Generator(flint, model, sequences, 160, int8) as gen:
            gen.prefill(u16(tokens[:, :prompt]))
            assert rel_l2(gen.logits().cpu(), want[:, prompt - 1]) <= 5e-3
            gen.step(u16(tokens[:, prompt]))
            assert rel_l2(gen.logits().cpu(), want[:, prompt]) <= 5e-3
    finally:
        model.close()
    assert not flint.kernel_fault()


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
@pytest.mark.parametrize("layers, sequences, heads", [(1, 64, 24), (2, 33, 20), (1, 33, 16), (1, 64, 12)])
def test_a_prompts_last_rows_run_on_what_a_step_runs_on(flint, layers, sequences, heads, int8):
    """Of many sequences of a wide FP16 model a step's linear layers run on the tensor-core GEMMs, with a LayerNorm
    launch of its own before MLP up; so do the prompt's last rows. The two last cases stay just below that."""
    cfg = dict(n_layer=layers, n_head=heads, n_embd=64 * heads, block_size=64, vocab_size=200, padded_vocab_size=208)
    params = weights(cfg)
    g = torch.Generator().manual_seed(11)
    tokens = torch.randint(0, 200, (sequences, 8), generator=g)
    want = oracle.gpt2_decode_logits(cfg, params, tokens, int8=int8)
    model = model_for(flint, cfg, params)
    launches = []
    try:
        for count in (1, sequences):
            with Generator(flint, model, count, 64, int8) as gen:
                before = flint.launch_count()
                gen.prefill(u16(tokens[:count]))
                launches.append(flint.launch_count() - before)
                assert rel_l2(gen.logits().cpu(), want[:count, 7]) <= 5e-3
    finally:
        model.close()
    assert launches[1] - launches[0] == (not int8 and sequences * 64 * heads >= 42000 and heads > 12)
    assert not flint.kernel_fault()


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
@pytest.mark.parametrize("sequences, heads, prompt", [(1, 2, 600), (20, 4, 8), (40, 4, 584), (2, 24, 24)])
def test_decode_kernels_at_their_edges_match_the_full_model(flint, sequences, heads, prompt, int8):
    """More positions than attention stages in shared memory; 17 to 32 and 33 to 64 rows of the
    linear kernels; the widest model; captured steps, whose kernels are resident several deep."""
    cfg = dict(n_layer=1, n_head=heads, n_embd=64 * heads, block_size=640, vocab_size=200, padded_vocab_size=208)
    params = weights(cfg)
    g = torch.Generator().manual_seed(5)
    tokens = torch.randint(0, 200, (sequences, prompt + 8), generator=g)
    want = oracle.gpt2_decode_logits(cfg, params, tokens, int8=int8)
    model = model_for(flint, cfg, params)
    try:
        with Generator(flint, model, sequences, 640, int8) as gen:
            gen.prefill(u16(tokens[:, :prompt]))
            for t in range(prompt, prompt + 8):
                chosen = gen.step(u16(tokens[:, t]), graph=t > prompt).cpu().to(torch.int64) & 0xFFFF
                got = gen.logits().cpu()
                assert rel_l2(got, want[:, t]) <= 5e-3, t
                assert torch.equal(chosen, got.argmax(1)), t
    finally:
        model.close()


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
@pytest.mark.parametrize("sequences, heads", [(12, 24), (24, 14), (40, 14), (33, 20), (64, 24)])
def test_wide_models_at_every_count_of_rows_match_the_full_model(flint, sequences, heads, int8):
    """Widths of 896 to 1,536 with 9 to 64 sequences: the linear kernels' longest shares of k, and
    normalised rows up to what shared memory holds (64 of 1,536: the sums then take their place)."""
    cfg = dict(n_layer=2, n_head=heads, n_embd=64 * heads, block_size=64, vocab_size=200, padded_vocab_size=208)
    params = weights(cfg)
    prompt, steps = 8, 4
    g = torch.Generator().manual_seed(8)
    tokens = torch.randint(0, 200, (sequences, prompt + steps), generator=g)
    want = oracle.gpt2_decode_logits(cfg, params, tokens, int8=int8)
    model = model_for(flint, cfg, params)
    try:
        with Generator(flint, model, sequences, 64, int8) as gen:
            gen.prefill(u16(tokens[:, :prompt]))
            assert rel_l2(gen.logits().cpu(), want[:, prompt - 1]) <= 5e-3
            for t in range(prompt, prompt + steps):
                chosen = gen.step(u16(tokens[:, t]), graph=t > prompt).cpu().to(torch.int64) & 0xFFFF
                got = gen.logits().cpu()
                assert rel_l2(got, want[:, t]) <= 5e-3, t
                assert torch.equal(chosen, got.argmax(1)), t
    finally:
        model.close()
    assert not flint.kernel_fault()


def teacher_forced_logits(flint, int8):
    """After a prompt and after each of six captured steps, of 8 sequences on six layers."""
    cfg = dict(n_layer=6, n_head=4, n_embd=256, block_size=320, vocab_size=200, padded_vocab_size=208)
    g = torch.Generator().manual_seed(9)
    tokens = torch.randint(0, 200, (8, 296 + 6), generator=g)
    model = model_for(flint, cfg, weights(cfg))
    try:
        with Generator(flint, model, 8, 320, int8) as gen:
            gen.prefill(u16(tokens[:, :296]))
            logits = [gen.logits().cpu()]
            for t in range(296, 302):
                gen.step(u16(tokens[:, t]), graph=True)
                logits.append(gen.logits().cpu())
    finally:
        model.close()
    return torch.stack(logits)


PLAIN_ORDER = """
import sys, numpy as np
sys.path[:0] = sys.argv[2:]
import flint_b200, test_generate_gpu as t
np.savez(sys.argv[1], *[t.teacher_forced_logits(flint_b200.Flint(), q).numpy() for q in (False, True)])
"""


def test_kernels_that_start_early_leave_what_plain_stream_order_leaves(flint, tmp_path):
    """A decode step's kernels are resident several deep and read ahead of their wait. In plain
    stream order (another process, FLINT_B200_PDL=0) nothing can be read too early: same bits."""
    root = Path(__file__).resolve().parent.parent
    out = tmp_path / "plain.npz"
    subprocess.run([sys.executable, "-c", PLAIN_ORDER, str(out), str(root / "tests"), str(root / "oracle"),
                    str(root)], check=True, env={**os.environ, "FLINT_B200_PDL": "0"}, timeout=300)
    plain = np.load(out)
    for i, int8 in enumerate((False, True)):
        assert np.array_equal(teacher_forced_logits(flint, int8).numpy(), plain[f"arr_{i}"])


@pytest.mark.parametrize("sequences", [1, 12, 40])
def test_logits_are_sums_in_fp32(flint, sequences):
    """A final LayerNorm of gain 0 leaves its bias, exactly: the logits are then dot products of
    known FP16 values, here 1,536 positive ones, whose FP32 sums show. Bound: 48 additions, each
    off by 2.4e-8 rms of what has been added up so far (1e-7 together), and 32 products added
    by the tensor core, cut at 2^-23 at worst (1.2e-7). A chain of 96 MMAs is off by over 1e-6."""
    cfg = dict(n_layer=1, n_head=24, n_embd=1536, block_size=64, vocab_size=200, padded_vocab_size=208)
    params = weights(cfg)
    g = torch.Generator().manual_seed(10)
    params["ln_f.weight"] = torch.zeros(1536)
    params["ln_f.bias"] = torch.randn(1536, generator=g).abs().half().float()
    params["wte.weight"] = (torch.randn(208, 1536, generator=g).abs() * 0.02).half().float()
    want = params["wte.weight"].double() @ params["ln_f.bias"].double()
    tokens = torch.randint(0, 200, (sequences, 9), generator=g)
    model = model_for(flint, cfg, params)
    try:
        with Generator(flint, model, sequences, 64, False) as gen:
            gen.prefill(u16(tokens[:, :8]))
            assert rel_l2(gen.logits().cpu(), want[:200].expand(sequences, -1)) <= 2.5e-7
            gen.step(u16(tokens[:, 8]))
            assert rel_l2(gen.logits().cpu(), want[:200].expand(sequences, -1)) <= 2.5e-7
    finally:
        model.close()


@pytest.mark.parametrize("int8", [False, True], ids=["fp16", "int8"])
def test_captured_steps_equal_plain_steps_bit_for_bit(flint, int8):
    params = weights(SMALL)
    g = torch.Generator().manual_seed(4)
    prompt = torch.randint(0, SMALL["vocab_size"], (4, 8), generator=g)
    model = model_for(flint, SMALL, params)
    try:
        runs = []
        for graph in (False, True):
            with Generator(flint, model, 4, 64, int8) as gen:
                chosen = gen.generate(u16(prompt), 20, graph=graph)
                runs.append((chosen, gen.logits().cpu()))
        assert torch.equal(runs[0][0], runs[1][0])
        assert torch.equal(runs[0][1], runs[1][1])
    finally:
        model.close()
    assert not flint.kernel_fault()


def test_gpt2_124m_decode_matches_the_full_model(flint):
    """GPT-2 124M, two sequences, a 64-token prompt and eight greedy steps: each step's logits
    against the oracle's on the sequence generated so far."""
    cfg = oracle.GPT2
    params = weights(cfg)
    g = torch.Generator().manual_seed(6)
    prompt = torch.randint(0, cfg["vocab_size"], (2, 64), generator=g)
    model = model_for(flint, cfg, params)
    try:
        with Generator(flint, model, 2, 128, False) as gen:
            chosen = gen.generate(u16(prompt), 9, graph=True)
            last = gen.logits().cpu()
        sequence = torch.cat([prompt, chosen[:, :8]], 1)             # 72 tokens
        want = oracle.gpt2_decode_logits(cfg, params, sequence)
        assert rel_l2(last, want[:, -1]) <= 5e-3
        # Each greedy choice is the oracle's, wherever the oracle's top two are not a near tie.
        for t in range(8):
            top = want[:, 63 + t].topk(2, dim=1)
            clear = (top.values[:, 0] - top.values[:, 1]) > 2e-2
            assert torch.equal(chosen[clear, t], top.indices[clear, 0]), t
    finally:
        model.close()
    assert not flint.kernel_fault()


def test_int8_copies_follow_the_stated_quantisation(flint):
    """The decoder's int8 path against the oracle's model with q * scale weights passes the
    same bound as FP16 (above); here the quantisation itself: weights that are already an
    int8 grid (up to their FP16 rounding) lose next to nothing when quantised again, so the
    int8 decoder follows the FP16 one far more closely than it would on arbitrary weights
    (about 2e-2 at these shapes)."""
    params = weights(SMALL)
    for name, p in params.items():
        if p.dim() == 2 and name != "wpe.weight":
            q, scale, approx = oracle.int8_rows(p)
            params[name] = approx.half().float() if name != "wte.weight" else p
    g = torch.Generator().manual_seed(7)
    tokens = torch.randint(0, SMALL["vocab_size"], (2, 16), generator=g)
    model = model_for(flint, SMALL, params)
    try:
        outs = []
        for int8 in (False, True):
            with Generator(flint, model, 2, 64, int8) as gen:
                gen.prefill(u16(tokens[:, :8]))
                for t in range(8, 16):
                    gen.step(u16(tokens[:, t]))
                outs.append(gen.logits().cpu())
        assert rel_l2(outs[1], outs[0]) <= 1e-2
    finally:
        model.close()


def test_generator_argument_errors(flint):
    params = weights(SMALL)
    model = model_for(flint, SMALL, params)
    try:
        import ctypes

        handle = ctypes.c_void_p(1)
        status = flint.lib.flint_b200_generator_create(model.handle, 0, 64, 0, ctypes.byref(handle))
        assert status == flint_b200.ERROR_INVALID_ARGUMENT and handle.value is None
        assert "sequences (0) must be from 1 to 64" in flint.last_error()
        status = flint.lib.flint_b200_generator_create(model.handle, 2, 60, 0, ctypes.byref(handle))
        assert status == flint_b200.ERROR_INVALID_ARGUMENT
        assert "max_length (60) must be a multiple of 8" in flint.last_error()
        with Generator(flint, model, 2, 16, False) as gen:
            with pytest.raises(flint_b200.FlintError, match="length .12. must be a multiple of 8"):
                gen.prefill(torch.zeros(2, 12, dtype=torch.int16, device=DEV))
            gen.prefill(torch.zeros(2, 16, dtype=torch.int16, device=DEV))
            with pytest.raises(flint_b200.FlintError, match="the cache is full"):
                gen.step(torch.zeros(2, dtype=torch.int16, device=DEV))
    finally:
        model.close()
