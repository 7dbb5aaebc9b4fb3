"""Model-level parity through the evo_* C ABI.

* Upstream's 50-layer tiny fixture (tests/golden/tiny, generated by upstream's
  tools/generate_tiny_model.py) against the logits of upstream's pure-Python
  BF16 oracle, with the tolerance of upstream's own CUDA model test
  (tests/test_cuda_model.cu:236-281: 0.08 abs + 0.06 rel, cosine >= 0.999).
* Mid-size fixtures (width 256, head size 128: every tensor-core and fused
  kernel is on the path) against upstream's CPU backend run through the same C
  ABI, with upstream's CPU-vs-CUDA profile gate (docs/execution-profiles.md:
  cosine >= 0.999, logit MAE <= 0.1, top-1 agreement >= 0.95).
"""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
TINY = ROOT / "tests" / "golden" / "tiny"
PROMPT = bytes([2, 5, 7, 3])
CHUNKED = bytes([2, 5, 7, 3, 9, 11, 13, 17, 19])
DECODE_TOKEN = 9


@pytest.fixture(scope="module")
def rt(pkg):
    import importlib

    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return importlib.import_module("evo_cpp_b200.runtime")


@pytest.fixture(scope="module")
def evo(rt, pkg):
    return rt.EvoLibrary(pkg.EVO_LIBRARY)


@pytest.fixture(scope="module")
def upstream_cpu(rt):
    path = ROOT / "oracle" / "_ref" / "libevo_ref.so"
    if not path.exists():
        pytest.skip("upstream CPU library was not built (make -C oracle ref)")
    return rt.EvoLibrary(path)


def close(actual, expected, atol, rtol, min_cosine=0.999):
    actual, expected = np.asarray(actual, np.float64).ravel(), np.asarray(expected, np.float64).ravel()
    assert actual.shape == expected.shape
    assert np.all(np.isfinite(actual))
    excess = np.abs(actual - expected) - (atol + rtol * np.abs(expected))
    assert excess.max() <= 0, excess.max()
    cosine = actual @ expected / (np.linalg.norm(actual) * np.linalg.norm(expected) + 1e-30)
    assert cosine >= min_cosine, cosine


def golden(name, columns):
    return np.fromfile(TINY / name, dtype="<f4").reshape(-1, columns)


def test_tiny_fixture_against_upstream_python_oracle(rt, evo):
    with pytest.raises(rt.EvoError) as refused:
        evo.load(TINY / "tiny.safetensors")
    assert refused.value.code == 5  # fixtures need the explicit test flag
    model = evo.load(TINY / "tiny.safetensors", flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    assert (model.vocab, model.width, model.layers) == (512, 8, 50)
    context = model.context(64)
    assert context.profile == "exact"
    logits = context.prefill(PROMPT)
    close(logits, golden("logits.f32", 512), 0.08, 0.06)
    assert context.position == 4
    step = context.decode(DECODE_TOKEN)
    close(step, golden("decode.f32", 512), 0.08, 0.06)
    assert context.position == 5
    # the fixture arena is 8 rows: 9 tokens run as an 8-row prefill + 1-row continuation
    chunked = model.context(64).prefill(CHUNKED)
    close(chunked, golden("chunked.f32", 512), 0.08, 0.06)
    layer = model.context(64).embed(PROMPT, 17)
    close(layer, golden("layer17.f32", 8), 0.08, 0.06)
    # two contexts of one model agree bit for bit; the model may be freed first
    other = model.context(64)
    model.close()
    assert np.array_equal(other.prefill(PROMPT), logits)
    with pytest.raises(rt.EvoError):
        other.prefill(PROMPT)  # prefill needs a fresh context
    with pytest.raises(rt.EvoError):
        model2 = evo.load(TINY / "tiny.safetensors", flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
        model2.context(64).embed(PROMPT, 50)  # layer out of range


def _fixture(tmp_path_factory, pkg, name, **kwargs):
    import importlib

    art = importlib.import_module("evo_cpp_b200.artifact")
    directory = tmp_path_factory.mktemp(name)
    spec = art.fixture_spec(**kwargs)
    art.write_synthetic(directory / "model.safetensors", spec, seed=3, weight_std=0.05, filter_std=0.3)
    return directory / "model.safetensors"


@pytest.fixture(scope="module")
def bf16_fixture(tmp_path_factory, pkg):
    return _fixture(tmp_path_factory, pkg, "bf16", width=256, layers=8, heads=2, inner=512,
                    hcs_groups=16, hcm_groups=16)


@pytest.fixture(scope="module")
def fp8_fixture(tmp_path_factory, pkg):
    return _fixture(tmp_path_factory, pkg, "fp8", width=256, layers=8, heads=2, inner=512,
                    hcs_groups=16, hcm_groups=16, fp8=True)


def _profile_gate(actual, expected):
    a, e = np.asarray(actual, np.float64), np.asarray(expected, np.float64)
    cosine = (a * e).sum() / (np.linalg.norm(a) * np.linalg.norm(e))
    mae = np.abs(a - e).mean()
    # Random-init logits are nearly flat, so top-1 is only meaningful where the
    # reference's winner leads by more than the rounding noise of a BF16 graph.
    ordered = np.sort(e, axis=-1)
    decided = (ordered[..., -1] - ordered[..., -2]) > 0.1
    agree = a.argmax(-1) == e.argmax(-1)
    top1 = agree[decided].mean() if decided.any() else 1.0
    overall = agree.mean() if agree.size >= 10 else 1.0
    assert cosine >= 0.999 and mae <= 0.1 and top1 >= 0.95 and overall >= 0.8, \
        (cosine, mae, top1, overall)


def test_bf16_fixture_against_upstream_cpu_backend(rt, evo, upstream_cpu, bf16_fixture):
    rng = np.random.default_rng(1000)
    sequence = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 40).tolist())
    reference_model = upstream_cpu.load(bf16_fixture, backend=rt.BACKEND_CPU,
                                        flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    reference_context = reference_model.context(128)
    expected = reference_context.prefill(sequence)
    model = evo.load(bf16_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    context = model.context(128)
    logits = context.prefill(sequence)          # 8-row arena: 5 chunks, continuation kernels
    assert logits.shape == expected.shape == (40, 512)
    _profile_gate(logits, expected)
    # greedy decode stays on upstream's trajectory
    sampler = rt.Sampler(evo)
    token = sampler.sample(logits[-1])
    for _ in range(6):
        step = context.decode(token)
        expected_step = reference_context.decode(token)
        _profile_gate(step[None], expected_step[None])
        token = sampler.sample(step)


def test_fp8_fixture_profiles_agree(rt, evo, fp8_fixture):
    """Bit-exact emulation profile vs tcgen05 profile on the same FP8 artifact:
    per-logit tolerance and identical top-1 on a seeded prompt."""
    rng = np.random.default_rng(1001)
    sequence = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 8).tolist())
    model = evo.load(fp8_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    exact = model.context(64)
    fast = model.context(64, flags=rt.CONTEXT_FLAG_TENSORCORE_FP8)
    assert (exact.profile, fast.profile) == ("exact", "b200-tc")
    a, b = exact.prefill(sequence), fast.prefill(sequence)
    # whole-model tolerance of upstream's CUDA model gate (0.08 abs + 0.06 rel)
    close(b, a, 0.08, 0.06)
    _profile_gate(b, a)
    # the emulation profile is deterministic across contexts
    assert np.array_equal(model.context(64).prefill(sequence), a)


def test_single_chunk_prefill_uses_fused_kernels_and_matches_chunked(rt, evo, upstream_cpu, bf16_fixture):
    """With the production arena the 300-token prompt is one chunk: fused
    projection-fed FIR / modal-scan kernels, flash attention, tcgen05 GEMMs."""
    rng = np.random.default_rng(1002)
    sequence = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 300).tolist())
    expected = upstream_cpu.load(bf16_fixture, backend=rt.BACKEND_CPU,
                                 flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC).context(512).prefill(sequence)
    model = evo.load(bf16_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    context = model.context(512, flags=rt.CONTEXT_FLAG_FULL_ARENA)
    logits = context.prefill(sequence)
    _profile_gate(logits, expected)
    chunked = model.context(512).prefill(sequence)   # 8-row chunks, continuation path
    _profile_gate(chunked, expected)
    _profile_gate(chunked, logits)
    # decode after the fused prefill continues from the caches it wrote
    reference_context = upstream_cpu.load(bf16_fixture, backend=rt.BACKEND_CPU,
                                          flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC).context(512)
    reference_context.prefill(sequence)
    token = int(logits[-1].argmax())
    for _ in range(4):
        step, expected_step = context.decode(token), reference_context.decode(token)
        _profile_gate(step[None], expected_step[None])
        token = int(step.argmax())


def _raw_prefill(rt, context, sequence, callback):
    """evo_context_prefill with a caller-supplied logits callback; returns the status."""
    batch = context._batch(bytes(sequence))
    try:
        return context.library.lib.evo_context_prefill(context.handle, batch, callback, None)
    finally:
        context.library.lib.evo_batch_free(batch)


def test_callback_errors_propagate_and_poison_the_context(rt, evo, bf16_fixture):
    """Upstream tests/test_cuda_c_api.c:100-194: a consumer that returns a non-OK status aborts the
    call with that status and the context refuses every later call; other contexts of the same
    model are untouched, and the model may be freed before them."""
    model = evo.load(bf16_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    first, second, third = model.context(64), model.context(64), model.context(64)
    model.close()                                   # contexts keep the weights alive
    sequence = b"ACGTACGTACGTACGTACGT"              # 20 tokens: three chunks of the 8-row fixture arena
    calls = []

    @rt.LOGITS_CALLBACK
    def fail_on_second_chunk(data, rows, cols, offset, _user):
        calls.append((rows, cols, offset))
        return 3 if len(calls) == 2 else 0          # EVO_STATUS_IO

    assert _raw_prefill(rt, first, sequence, fail_on_second_chunk) == 3
    assert calls == [(8, 512, 0), (8, 512, 8)]
    assert b"io: " in evo.lib.evo_last_error()
    with pytest.raises(rt.EvoError) as poisoned:
        first.decode(65)
    assert poisoned.value.code == 2 and "invalidated" in str(poisoned.value)
    with pytest.raises(rt.EvoError):
        first.prefill(sequence)
    # a status outside the enum is reported as internal
    @rt.LOGITS_CALLBACK
    def nonsense(data, rows, cols, offset, _user):
        return 12345

    assert _raw_prefill(rt, second, sequence, nonsense) == 70
    # decode: the callback's error poisons as well
    expected = third.prefill(sequence)
    assert expected.shape == (20, 512)

    @rt.LOGITS_CALLBACK
    def refuse(data, rows, cols, offset, _user):
        return 5

    assert evo.lib.evo_context_decode(third.handle, 65, refuse, None) == 5
    with pytest.raises(rt.EvoError) as poisoned:
        third.decode(65)
    assert poisoned.value.code == 2


def test_invalid_precision_metadata_is_rejected_with_upstreams_messages(rt, evo, pkg, tmp_path):
    """Upstream tests/test_cuda_model.cu:195-208 (messages from src/cuda/model.cu:711-724, 991-997)."""
    import importlib

    art = importlib.import_module("evo_cpp_b200.artifact")
    base = dict(width=64, layers=4, heads=1, inner=128, hcs_groups=8, hcm_groups=8)

    def write(name, mutate, extra=None):
        spec = art.fixture_spec(**base)
        mutate(spec)
        tensors = list(art.synthetic_tensors(spec, seed=1))
        if extra is not None:
            tensors.append(extra)
        path = tmp_path / f"{name}.safetensors"
        art.write_model(path, spec["metadata"], tensors)
        return path

    def expect(path, code, fragment):
        with pytest.raises(rt.EvoError) as refused:
            evo.load(path, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
        assert refused.value.code == code and fragment in str(refused.value), str(refused.value)

    expect(write("disagrees", lambda s: s["metadata"].update({"hyena_projection_dtype": art.typed("E4M3_SW")})),
           4, "disagrees")
    expect(write("dtype", lambda s: s["metadata"].update({"hyena_projection_dtype": art.typed("INT8")})),
           5, "unsupported Hyena projection dtype: INT8")
    expect(write("extra", lambda s: None, ("blocks.0.surplus", "F32", [4], bytes(16))), 4,
           "unknown tensor for model profile")


def test_cached_prefill_refuses_chunk_continuation_and_bad_device_tokens_are_caught(rt, evo, bf16_fixture):
    import torch

    model = evo.load(bf16_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    context = model.context(64)
    # upstream tests/test_cuda_model.cu:283-292: after the exact cached-attention prefill only
    # token decode may continue the sequence
    logits, _ = context.prefill_with_dumps(b"AC", [], cached=True)
    assert logits.shape == (2, 512)
    tokens = torch.tensor([71], dtype=torch.int32, device="cuda")
    with pytest.raises(rt.EvoError) as refused:
        context.continue_device(tokens.data_ptr(), 1)
    assert refused.value.code == 2 and "cached prefill" in str(refused.value)
    assert context.decode(71).shape == (512,)
    # a device-resident id outside the vocabulary is never used as a table index: the pass is
    # reported as an invalid argument at the next synchronisation and the context is retired
    context = model.context(64)
    tokens = torch.tensor([65, 67, 9999, 71], dtype=torch.int32, device="cuda")
    context.prefill_device(tokens.data_ptr(), 4, stateless=True)
    with pytest.raises(rt.EvoError) as bad:
        context.synchronize()
    assert bad.value.code == 2 and "vocabulary" in str(bad.value)
    with pytest.raises(rt.EvoError):
        context.prefill(b"ACGT")


def test_prefill_forms_on_token_ids(rt, evo):
    """evo_b200_context_prefill_tokens, the forms of upstream's model classes (include/evo/cuda/model.hpp:121-170)
    on the tiny fixture: FRESH equals evo_context_prefill and may be repeated on a used context, STATELESS gives the
    same bits and leaves position 0 (decode refused after it), CHUNK continues a FRESH prefill, CACHED continues
    through decode only (upstream tests/test_cuda_model.cu:196-292)."""
    model = evo.load(TINY / "tiny.safetensors", flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    context, other = model.context(12), model.context(12)
    assert context.activation_capacity == 8
    prompt = [2, 5, 7, 3]
    reference = other.prefill(bytes(prompt))
    assert np.array_equal(context.prefill_tokens([1]), other_first := model.context(12).prefill(bytes([1])))
    assert context.position == 1 and other_first.shape == (1, 512)
    stateless = context.prefill_tokens(prompt, context.PREFILL_STATELESS)
    assert context.position == 0 and np.array_equal(stateless, reference)
    with pytest.raises(rt.EvoError):
        context.decode(9)
    fresh = context.prefill_tokens(prompt)                      # the refused decode did not retire the context
    assert context.position == 4 and np.array_equal(fresh, reference)
    assert np.array_equal(context.decode(9), other.decode(9))
    long_prompt = [2, 5, 7, 3, 9, 11, 13, 17, 19]
    context.prefill_tokens(long_prompt[:8])
    last = context.prefill_tokens(long_prompt[8:], context.PREFILL_CHUNK)
    whole = model.context(12).prefill(bytes(long_prompt))       # the portable entry chunks by itself
    assert context.position == 9 and np.array_equal(last[0], whole[8])
    with pytest.raises(rt.EvoError):                            # more than one activation chunk
        context.prefill_tokens(long_prompt, context.PREFILL_STATELESS)
    # embeddings chunk by chunk on token ids equal the portable entry's rows (it chunks by itself)
    expected_rows = model.context(12).embed(bytes(long_prompt), 17)
    first_rows = context.embed_tokens(long_prompt[:8], 17)
    last_rows = context.embed_tokens(long_prompt[8:], 17, first_chunk=False)
    assert context.position == 9 and np.array_equal(np.concatenate([first_rows, last_rows]), expected_rows)
    with pytest.raises(rt.EvoError):
        context.embed_tokens([2], 50)
    cached = context.prefill_tokens([2, 5], context.PREFILL_CACHED)
    assert cached.shape == (2, 512) and context.position == 2
    with pytest.raises(rt.EvoError) as refused:
        context.prefill_tokens([7], context.PREFILL_CHUNK)
    assert "exact token decode" in str(refused.value)
    assert context.decode(7).shape == (512,)


def test_embedding_is_chunked_and_advances_the_context_like_upstream(rt, evo, bf16_fixture):
    """Upstream src/c_api.cpp:1075-1330: a fresh context, one callback per activation chunk with its token
    offset, the position advanced; the rows equal a single-chunk capture up to the continuation kernels'
    summation order; a failing consumer invalidates the context."""
    model = evo.load(bf16_fixture, flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC)
    rng = np.random.default_rng(77)
    sequence = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 21).tolist())
    context = model.context(64)                                        # 8-row arena: chunks of 8, 8 and 5 rows
    offsets = []

    @rt.LOGITS_CALLBACK
    def record(data, rows, cols, offset, _user):
        offsets.append((rows, cols, offset))
        return 0

    batch = context._batch(sequence)
    assert evo.lib.evo_context_embed(context.handle, batch, 5, record, None) == 0
    evo.lib.evo_batch_free(batch)
    assert offsets == [(8, 256, 0), (8, 256, 8), (5, 256, 16)] and context.position == 21
    with pytest.raises(rt.EvoError) as used:
        context.embed(sequence, 5)                                     # needs a fresh context
    assert used.value.code == 2 and "fresh context" in str(used.value)
    chunked = model.context(64).embed(sequence, 5)
    whole = model.context(64, flags=rt.CONTEXT_FLAG_FULL_ARENA).embed(sequence, 5)
    assert chunked.shape == whole.shape == (21, 256)
    close(chunked, whole, 0.08, 0.06)

    @rt.LOGITS_CALLBACK
    def refuse(data, rows, cols, offset, _user):
        return 3

    failing = model.context(64)
    batch = failing._batch(sequence)
    assert evo.lib.evo_context_embed(failing.handle, batch, 5, refuse, None) == 3
    evo.lib.evo_batch_free(batch)
    with pytest.raises(rt.EvoError):
        failing.prefill(sequence)


@pytest.mark.parametrize("limit", [0, 4096])
@pytest.mark.parametrize("decoder", [False, True], ids=["stripedhyena", "decoder"])
def test_results_without_pinned_memory(rt, evo, pkg, fp8_fixture, tmp_path, monkeypatch, decoder, limit):
    """Contexts need no pinned memory: without any, or with results above the limit, logits come back through pageable
    copies (BF16 ones are widened in place), bit for bit the same, and errors are still reported."""
    if decoder:
        from gigusun_util import attention, delta, gla, make_model

        path, flags = make_model(pkg, tmp_path / "m", [delta(), attention(), gla()])[0], 0
    else:
        path, flags = fp8_fixture, rt.MODEL_FLAG_ALLOW_SYNTHETIC
    usual = evo.load(path, flags=flags)
    monkeypatch.setenv("EVO_B200_PINNED_BYTES", str(limit))
    limited = evo.load(path, flags=flags)
    monkeypatch.delenv("EVO_B200_PINNED_BYTES")
    tokens = np.random.default_rng(3).integers(0, usual.vocab, 150).tolist()
    full = 0 if decoder else rt.CONTEXT_FLAG_FULL_ARENA
    a, b = usual.context(256, full), limited.context(256, full)
    for prompt in (tokens[:1], tokens[:7], tokens):
        assert np.array_equal(a.prefill_tokens(prompt), b.prefill_tokens(prompt))
    for token in tokens[:5]:
        assert np.array_equal(a.decode(token), b.decode(token))
    assert np.array_equal(a.embed_tokens(tokens[:20], 1), b.embed_tokens(tokens[:20], 1))
    for context in (a, b):
        with pytest.raises(rt.EvoError) as refused:
            context.prefill_tokens([0, usual.vocab])
        assert refused.value.code == 2
    for closed in (a, b, usual, limited):
        closed.close()
