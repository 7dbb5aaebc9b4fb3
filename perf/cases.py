"""What the framework's speed is measured on: prompts and generation through the model-level API.

Four models stand for the shapes that this repository's configurations and benchmark use, with fewer blocks and
random weights of the checkpoints' types: StripedHyena2 at the width of evo2_7b and of evo2_1b_base (every mixer,
E4M3 Hyena projections), and the two decoder designs at the width 2,048 of the benchmark.  A pass is what a program
does with a context that it keeps: a prompt to logits (token ids on the host, F32 logits back on the host, or
resident on the device), or a prompt followed by single-token steps.  Steps are fed given tokens, so that a near
tie of two logits cannot send two correct implementations along different sequences.

The weights of a model are one seeded file per machine, written on first use and loaded once per process; the
tokens of a case come from its seed.  exact() reads the same file and computes the logits in float64.
"""
from __future__ import annotations

import importlib
import importlib.util
import json
import math
import os
import shutil
import struct
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path.cwd()
PACKAGE = "evo_cpp_b200"

VOCAB = 512
MAX_TOKENS = 8192  # rows of the activation arena: the longest prompt that one pass takes
WINDOW, KEEP = 1024, 4

# StripedHyena2 blocks cycle short, medium and long convolution and attention.  1,920 channels in 128 filter groups
# and 15 heads (evo2_1b_base), 4,096 in 256 groups and 32 heads (evo2_7b).
HYENA = {
    "hyena-1920": dict(width=1920, layers=8, heads=15, inner=5120, hcs_groups=128, hcm_groups=128),
    "hyena-4096": dict(width=4096, layers=4, heads=32, inner=11264, hcs_groups=256, hcm_groups=256),
}
DECODERS = ("gigusun-2048", "kikepel-2048")

FORMAT = 1  # of the weight files: part of their path


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a short query on the smallest model: launches and host calls are what counts
        dict(name="hyena1920-short", model="hyena-1920", kind="generate", tokens=19, steps=3, profile="b200-tc"),
        # sequence scoring with a length that is a multiple of nothing, host to host
        dict(name="hyena1920-score", model="hyena-1920", kind="prefill", tokens=3001, steps=0, profile="b200-tc"),
        # the default profile: generation behind a gene-sized prompt
        dict(name="hyena4096-generate-exact", model="hyena-4096", kind="generate", tokens=200, steps=32, profile="exact"),
        # the default profile: scoring of a variant window
        dict(name="hyena4096-score-exact", model="hyena-4096", kind="prefill", tokens=509, steps=0, profile="exact"),
        # a few tokens: a stream of the weights
        dict(name="hyena4096-few", model="hyena-4096", kind="prefill", tokens=61, steps=0, profile="b200-tc"),
        dict(name="hyena4096-score", model="hyena-4096", kind="prefill", tokens=1000, steps=0, profile="b200-tc"),
        # the headline workload: the longest prompt of one pass, tokens and logits on the device
        dict(name="hyena4096-prompt", model="hyena-4096", kind="device", tokens=8192, steps=0, profile="b200-tc"),
        # step after step on a decoder with attention and matrix states
        dict(name="gigusun-generate", model="gigusun-2048", kind="generate", tokens=150, steps=48, profile="exact"),
        # trace replay in the F32 profile
        dict(name="gigusun-replay-f32", model="gigusun-2048", kind="generate", tokens=90, steps=16, profile="float32"),
        dict(name="gigusun-prompt", model="gigusun-2048", kind="device", tokens=8192, steps=0, profile="exact"),
        # latents and experts: step after step, and a prompt of an odd length
        dict(name="kikepel-generate", model="kikepel-2048", kind="generate", tokens=100, steps=48, profile="exact"),
        dict(name="kikepel-score", model="kikepel-2048", kind="prefill", tokens=2999, steps=0, profile="exact"),
    ]


def draw(rng):
    """A model, a kind of pass and a profile of the listed ones; lengths spread over their logarithm.  The profiles
    that compute on the CUDA cores get shorter prompts, as they do in use."""
    model = rng.choice(sorted(HYENA) + list(DECODERS))
    kind = rng.choice(("prefill", "device", "generate", "generate"))
    slow = rng.random() < 0.3
    profile = ("exact" if slow else "b200-tc") if model in HYENA else ("float32" if slow else "exact")
    longest = 1000 if kind == "generate" else MAX_TOKENS
    if slow:
        longest = {"hyena-4096": 509, "hyena-1920": 1200}.get(model, 160)
        if kind == "generate":
            longest = {"hyena-4096": 220, "hyena-1920": 500}.get(model, longest)
    tokens = min(longest, int(round(math.exp(rng.uniform(math.log(9), math.log(longest))))))
    steps = int(round(math.exp(rng.uniform(0.0, math.log(32 if slow else 48))))) if kind == "generate" else 0
    return dict(model=model, kind=kind, tokens=tokens, steps=steps, profile=profile)


# ------------------------------------------------------------------------------------------------ models
def package():
    if PACKAGE not in sys.modules:
        directory = ROOT / "evo.cpp_b200"
        spec = importlib.util.spec_from_file_location(PACKAGE, directory / "__init__.py",
                                                      submodule_search_locations=[str(directory)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[PACKAGE] = module
        spec.loader.exec_module(module)
    return sys.modules[PACKAGE]


def part(name):
    package()
    return importlib.import_module(f"{PACKAGE}.{name}")


def decoder_config(model):
    heads, width = 16, 2048
    if model == "gigusun-2048":
        mlp = {"kind": "dense", "ff": 8448}
        delta = {"type": "delta", "mlp": mlp,
                 "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
        attention = {"type": "attention", "mlp": mlp,
                     "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                               "softcap": 30.0, "mask": {"size": WINDOW, "keep_first": KEEP}}}
        gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": heads // 2, "dim": 128, "vdim": 256, "tau": 16.0}}
        return part("artifact").gigusun_config([delta, attention, gla] * 2, vocab=VOCAB, width=width,
                                               max_positions=MAX_TOKENS + 64)
    layers = []
    for i in range(4):
        mlp = {"kind": "dense", "ff": 5632} if i == 0 else {
            "kind": "moe", "expert": {"ff": 1408, "limit": 7.0}, "router": {"experts": 32, "top": 4}}
        layers.append({"type": ("latent_attention", "latent_attention_2")[i % 2], "mlp": mlp,
                       "mixer": {"heads": heads, "dim": 128, "vdim": 128, "q_rank": 768, "kv_rank": 512,
                                 "scale": 128 ** -0.5, "mask": {"size": WINDOW}}})
    return part("artifact").kikepel_config(layers, vocab=VOCAB, width=width)


def damp_experts(directory, config):
    """Gains of 1/8 behind the mixtures of experts.  A random router has near ties: two correct implementations send
    a few rows to different experts, and with gains around one these rows would be all that a comparison sees."""
    path = directory / "model.safetensors"
    with open(path, "rb") as file:
        length = struct.unpack("<Q", file.read(8))[0]
        header = json.loads(file.read(length))
    for i, layer in enumerate(config["layers"]):
        if layer["mlp"]["kind"] == "moe":
            begin, end = header[f"l{i}.norm2"]["data_offsets"]
            stored = np.memmap(path, np.uint16, "r+", 8 + length + begin, (end - begin) // 2)
            stored -= np.uint16(3 << 7)  # the exponent of a BF16 value, three lower
            stored.flush()


def weights_path(model):
    """The model's file (StripedHyena2) or directory (decoders); written if this machine has none yet."""
    base = Path(tempfile.gettempdir()) / f"evo_b200_perf_{os.getuid()}_{FORMAT}"
    directory = base / model
    if not (directory / "COMPLETE").exists():
        base.mkdir(parents=True, exist_ok=True)
        fresh = Path(tempfile.mkdtemp(prefix=model, dir=base))
        art = part("artifact")
        if model in HYENA:
            spec = art.fixture_spec(fp8=True, vocab=VOCAB, **HYENA[model])
            art.write_synthetic(fresh / "model.safetensors", spec, 1, filter_std=0.1, device="cuda", max_shard_bytes=1 << 40)
        else:
            art.write_decoder_random(fresh, decoder_config(model), 5, "cuda")
            damp_experts(fresh, decoder_config(model))
        (fresh / "COMPLETE").write_text("ok\n")
        try:
            fresh.rename(directory)
        except OSError:  # another process was first
            shutil.rmtree(fresh, ignore_errors=True)
    return directory / "model.safetensors" if model in HYENA else directory


LOADED = {}


def loaded(model):
    if model not in LOADED:
        rt = part("runtime")
        library = rt.EvoLibrary(package().EVO_LIBRARY)
        LOADED[model] = library.load(weights_path(model), flags=rt.MODEL_FLAG_ALLOW_SYNTHETIC if model in HYENA else 0)
    return LOADED[model]


def flags(case):
    rt = part("runtime")
    value = {"exact": 0, "b200-tc": rt.CONTEXT_FLAG_TENSORCORE_FP8, "float32": rt.CONTEXT_FLAG_FLOAT32}[case["profile"]]
    return value | (rt.CONTEXT_FLAG_FULL_ARENA if case["model"] in HYENA else 0)


def token_ids(case, seed):
    rng = np.random.default_rng(seed)
    count = case["tokens"] + case["steps"]
    if case["model"] in HYENA:
        return rng.choice(np.frombuffer(b"ACGT", np.uint8), count).astype(np.int64)
    return rng.integers(0, VOCAB, count)


# ------------------------------------------------------------------------------------------------ a pass
class DeviceLogits:
    """Logits in the context's own buffer: BF16 for StripedHyena2, F32 for decoders.  A tensor made from this keeps it,
    and with it the context, alive."""

    def __init__(self, address, rows, hyena, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (rows, VOCAB), "typestr": "<i2" if hyena else "<f4",
                                         "data": (address, False), "version": 2, "strides": None}


class State:
    def __init__(self, case, seed):
        self.case = case
        self.context = None
        ids = token_ids(case, seed)
        self.prompt, self.steps = [int(t) for t in ids[:case["tokens"]]], [int(t) for t in ids[case["tokens"]:]]
        self.device_tokens = torch.from_numpy(ids[:case["tokens"]].astype(np.int32)).cuda() if case["kind"] == "device" else None
        self.context = loaded(case["model"]).context(case["tokens"] + case["steps"], flags(case))

    def __del__(self):
        if self.context is not None:
            self.context.close()


def prepare(case, seed):
    return State(case, seed)


def run(state):
    case, context = state.case, state.context
    if case["kind"] == "device":
        address = context.prefill_device(state.device_tokens.data_ptr(), case["tokens"], True)
        hyena = case["model"] in HYENA
        logits = torch.as_tensor(DeviceLogits(address, case["tokens"], hyena, state), device="cuda")
        return logits.view(torch.bfloat16) if hyena else logits
    prompt = context.prefill_tokens(state.prompt)
    if case["kind"] == "prefill":
        return prompt
    return {"prompt": prompt, "steps": np.stack([context.decode(token) for token in state.steps])}


# ------------------------------------------------------------------------------------------------ work and tolerance
def seen_keys(begin, rows, window=None, keep=0):
    """Pairs of a query in [begin, begin + rows) and a key that it sees."""
    i = np.arange(begin, begin + rows, dtype=np.float64) + 1
    return float(i.sum() if window is None else (np.minimum(i, window) + np.clip(i - window, 0, keep)).sum())


def pass_work(case, begin, rows):
    """(bytes, FLOPs) of `rows` tokens behind `begin` earlier ones: every weight, token and cached key once, logits out."""
    wide = 4.0 if case["kind"] != "device" or case["model"] not in HYENA else 2.0
    nbytes, flops = rows * (4.0 + VOCAB * wide), 2.0 * rows * VOCAB
    if case["model"] in HYENA:
        s = HYENA[case["model"]]
        D, inner, layers = s["width"], s["inner"], s["layers"]
        quarter = layers // 4
        matrices = layers * (4.0 * D * D + 3.0 * D * inner) + VOCAB * D
        nbytes += 2.0 * matrices - 3.0 * quarter * 3.0 * D * D  # one byte per weight of the Hyena projections
        flops = 2.0 * rows * matrices + quarter * (4.0 * D * seen_keys(begin, rows) + 2.0 * rows * D * (9 + 7 + 128 + 48))
        nbytes += quarter * 4.0 * D * begin
        return nbytes, flops
    config = decoder_config(case["model"])
    D = config["width"]
    weights = VOCAB * D
    active = float(weights)
    for layer in config["layers"]:
        m, mlp = layer["mixer"], layer["mlp"]
        H, dim, vdim = m["heads"], m["dim"], m["vdim"]
        if "kv_rank" in m:
            q, c = m["q_rank"], m["kv_rank"]
            matrices = (q + c) * D + q * H * dim + c * H * (dim + vdim) + D * H * vdim
            flops += 2.0 * H * (dim + vdim) * seen_keys(begin, rows, WINDOW)
            nbytes += 2.0 * c * min(begin, WINDOW)
        elif layer["type"] == "attention":
            G = m["kv_heads"]
            matrices = ((H + G) * dim + G * vdim + H) * D + D * H * vdim
            flops += 2.0 * H * (dim + vdim) * seen_keys(begin, rows, WINDOW, KEEP)
            nbytes += 2.0 * G * (dim + vdim) * min(begin, WINDOW + KEEP)
        else:
            G = m.get("kv_heads", H)
            matrices = (2 * G * dim + 2 * H * vdim) * D + D * H * vdim
            flops += 8.0 * rows * H * dim * vdim
            nbytes += 8.0 * H * dim * vdim if begin else 4.0 * H * dim * vdim
        weights += matrices
        active += matrices
        if mlp["kind"] == "moe":
            one = 3.0 * D * mlp["expert"]["ff"]
            experts, top = mlp["router"]["experts"], mlp["router"]["top"]
            weights += experts * D + one * min(experts, rows * top)
            active += experts * D + one * top
        else:
            one = (2.0 if case["model"] == "gigusun-2048" else 3.0) * D * mlp["ff"]
            weights += one
            active += one
    return nbytes + 2.0 * weights, flops + 2.0 * rows * active


def work(case):
    nbytes, flops = pass_work(case, 0, case["tokens"])
    for i in range(case["steps"]):
        more = pass_work(case, case["tokens"] + i, 1)
        nbytes, flops = nbytes + more[0], flops + more[1]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Logits behind a stack of blocks.  With BF16 activations a sum in another order turns some roundings of every
    layer the other way: 0.016 to 0.023 (StripedHyena2), 0.007 (Gigusun) and 0.01 (Kikepel, where a few rows also meet
    another expert) from float64; 1e-6 in F32."""
    if case["profile"] == "float32":
        return {"rel": 5e-6, "max": 1e-4}
    return {"rel": 0.02 if case["model"] == "gigusun-2048" else 0.03, "max": 0.5}


# ------------------------------------------------------------------------------------------------ the same in float64
def read_weights(path):
    """{name: tensor on the GPU in its stored type} of a Safetensors file."""
    data = np.memmap(path, np.uint8, "r")
    length = struct.unpack("<Q", bytes(data[:8]))[0]
    header = json.loads(bytes(data[8:8 + length]))
    types = {"F32": torch.float32, "BF16": torch.bfloat16, "F8_E4M3": torch.float8_e4m3fn}
    found = {}
    for name, entry in header.items():
        if name == "__metadata__":
            continue
        begin, end = entry["data_offsets"]
        raw = torch.from_numpy(np.array(data[8 + length + begin:8 + length + end])).cuda()
        found[name] = raw.view(types[entry["dtype"]]).reshape(entry["shape"])
    return found


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def softmax_attention(q, k, v, scale, bias=None, window=None, keep=0, softcap=0.0, sink=None):
    """q, k [T, H, dim], v [T, H, vdim]; bias(head) -> [T] added by distance; sink: None or [H] logits without a value."""
    T, H = q.shape[:2]
    i = torch.arange(T, device=q.device)
    distance = i[:, None] - i[None, :]
    hidden = distance < 0
    if window is not None:
        hidden |= (distance >= window) & (i[None, :] >= keep)
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = q[:, h] @ k[:, h].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if bias is not None:
            s = s - bias(h)[distance.clamp(min=0)]
        s = s.masked_fill(hidden, -math.inf)
        top = s.amax(-1, keepdim=True) if sink is None else torch.maximum(s.amax(-1, keepdim=True), sink[h])
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out[:, h] = e @ v[:, h] / total
    return out


def causal_fir(x, taps, newest_last):
    """x [T, C], taps [C, n]; the last (or the first) tap meets the current row."""
    T, n = len(x), taps.shape[1]
    y = torch.zeros_like(x)
    for j in range(min(n, T)):
        y[j:] += x[:T - j] * taps[:, n - 1 - j if newest_last else j]
    return y


def long_convolution(x, h):
    """Causal convolution of x and h [T, C] through an FFT of twice the length."""
    n = 2 * len(x)
    y = torch.empty_like(x)
    for c in range(0, x.shape[1], 256):
        y[:, c:c + 256] = torch.fft.irfft(torch.fft.rfft(x[:, c:c + 256], n, 0) * torch.fft.rfft(h[:, c:c + 256], n, 0),
                                          n, 0)[:len(x)]
    return y


def hyena_logits(model, ids):
    s, w = HYENA[model], read_weights(weights_path(model))
    D, heads, T = s["width"], s["heads"], len(ids)

    def norm(x, name):
        return x / (torch.sqrt((x * x).mean(-1, keepdim=True)) + 1e-6) * w[name].double()

    x = w["embedding_layer.weight"].double()[ids]
    for i in range(s["layers"]):
        p, kind = f"blocks.{i}.", i % 4
        h = norm(x, p + "pre_norm.scale")
        if kind == 3:
            d = D // heads
            qkv = (h @ w[p + "inner_mha_cls.Wqkv.weight"].double().T).reshape(T, 3, heads, d)
            angle = torch.arange(T, device=x.device)[:, None] * w[p + "inner_mha_cls.rotary_emb.inv_freq"].double()
            cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

            def rotate(t):
                a, b = t[..., :d // 2], t[..., d // 2:]
                return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

            mixed = softmax_attention(rotate(qkv[:, 0]), rotate(qkv[:, 1]), qkv[:, 2], d ** -0.5).reshape(T, D)
            out = "inner_mha_cls.out_proj."
        else:
            scales = w[p + "projections.fp8_runtime_scales"].double()
            codes = (h.bfloat16().double() * scales[0]).clamp(-448, 448).float().to(torch.float8_e4m3fn).double()
            z = codes @ w[p + "projections.weight"].double().T * scales[1]
            z = causal_fir(z, w[p + "filter.short_filter_weight"].double().reshape(3 * D, 3), True).reshape(T, D, 3)
            u = z[..., 1] * z[..., 2]
            if kind == 2:
                t = torch.arange(T, device=x.device, dtype=torch.float64)
                poles, residues = w[p + "filter.log_poles"].double()[..., 0], w[p + "filter.residues"].double()
                kernel = sum(residues[:, m] * torch.exp(t[:, None] * poles[:, m]) for m in range(poles.shape[1]))
                y = long_convolution(u, kernel) + u * w[p + "filter.D"].double()
            else:
                taps = w[p + "filter.h"].double()[:, 0]
                taps = taps.repeat_interleave(D // len(taps), 0)
                y = causal_fir(u, taps, kind == 0)
                if kind == 1:
                    y = y + u * w[p + "filter.D"].double()
            mixed = y * z[..., 0]
            out = "out_filter_dense."
        x = x + mixed @ w[p + out + "weight"].double().T + w[p + out + "bias"].double()
        h = norm(x, p + "post_norm.scale")
        a = h @ w[p + "mlp.l1.weight"].double().T
        if i == 0:
            a = torch.nn.functional.gelu(a)
        x = x + (a * (h @ w[p + "mlp.l2.weight"].double().T)) @ w[p + "mlp.l3.weight"].double().T
    return norm(x, "norm.scale") @ w["embedding_layer.weight"].double().T


def gated_linear(h, w, p, m):
    T, H = len(h), m["heads"]
    q = (h @ w(p + "q").T).reshape(T, H, m["dim"]) * m["dim"] ** -0.5
    k = (h @ w(p + "k").T).reshape(T, H, m["dim"])
    v = (h @ w(p + "v").T).reshape(T, H, m["vdim"])
    decay = (h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "a2.b")
    decay = torch.exp(-torch.nn.functional.softplus(-decay) / m["tau"]).reshape(T, H, m["dim"])
    state = torch.zeros(H, m["dim"], m["vdim"], dtype=h.dtype, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        state = torch.baddbmm(state * decay[t][:, :, None], k[t][:, :, None], v[t][:, None, :])
        out[t] = torch.bmm(q[t][:, None, :], state)[:, 0]
    return (rms(out, 1e-6) * w(p + "norm")).reshape(T, -1) * silu(h @ w(p + "g").T)


def gated_delta(h, w, p, m):
    T, H, G = len(h), m["heads"], m["kv_heads"]
    q, k, v = (silu(causal_fir(h @ w(p + n).T, w(p + n + ".conv"), True)) for n in "qkv")

    def unit(x):
        x = x.reshape(T, G, m["dim"])
        return (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)

    q, k, v = unit(q) * m["dim"] ** -0.5, unit(k), v.reshape(T, H, m["vdim"])
    beta = torch.sigmoid(h @ w(p + "b").T)
    decay = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").T + w(p + "dt_bias")))
    state = torch.zeros(H, m["dim"], m["vdim"], dtype=h.dtype, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        state = state * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], state)[:, 0])
        state = torch.baddbmm(state, k[t][:, :, None], u[:, None, :])
        out[t] = torch.bmm(q[t][:, None, :], state)[:, 0]
    out = rms(out, 1e-6) * w(p + "norm")
    return out.reshape(T, -1) * silu(h @ w(p + "g").T)


def gigusun_logits(ids):
    config, stored = decoder_config("gigusun-2048"), read_weights(weights_path("gigusun-2048") / "model.safetensors")
    eps, T = config["norm"]["eps"], len(ids)

    def w(name):
        return stored[name].double()

    def norm(x, name):
        return rms(x, eps) * (1.0 + w(name))

    x = norm(w("embed")[ids] + w("pos")[:T], "embed.norm")
    for i, layer in enumerate(config["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        h = norm(x, f"l{i}.norm1")
        if layer["type"] == "attention":
            H, G = m["heads"], m["kv_heads"]
            q = rms((h @ w(p + "q").T).reshape(T, H, m["dim"]), eps) * w(p + "q.norm")
            k = rms((h @ w(p + "k").T).reshape(T, G, m["dim"]), eps) * w(p + "k.norm")
            v = (h @ w(p + "v").T).reshape(T, G, m["vdim"])
            far = torch.arange(T, device=x.device, dtype=torch.float64)
            r1, r2 = w(p + "r1"), w(p + "r2")
            o = softmax_attention(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), m["scale"],
                                  lambda head: r1[head] * torch.log1p(r2[head] * far), m["mask"]["size"],
                                  m["mask"]["keep_first"], m["softcap"], torch.zeros(H, dtype=x.dtype, device=x.device))
            o = (o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(T, -1)
        else:
            o = (gated_linear if layer["type"] == "gla" else gated_delta)(h, w, p, m)
        x = x + o @ w(p + "o").T
        z = norm(x, f"l{i}.norm2") @ w(f"l{i}.mlp.up").T
        a, b, c, e = w(f"l{i}.mlp.act")
        x = x + (a * rms(z, eps) + b * rms(z ** 2, eps) + c * rms(z ** 3, eps) + e) @ w(f"l{i}.mlp.down").T
    return norm(x, "final.norm") @ w("head").T


def mixture(h, w, p, mlp):
    scores = torch.sigmoid(h @ w(p + "router").T)
    weight, chosen = torch.topk(scores, mlp["router"]["top"], dim=-1)
    limit, out = mlp["expert"]["limit"], torch.zeros_like(h)
    for e in range(scores.shape[1]):
        row, slot = torch.nonzero(chosen == e, as_tuple=True)
        inner = h[row] * weight[row, slot][:, None]
        g = torch.clamp(inner @ w(f"{p}e{e}.gate").T, max=limit)
        u = torch.clamp(inner @ w(f"{p}e{e}.up").T, -limit, limit)
        out.index_add_(0, row, (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"{p}e{e}.down").T)
    return out


def kikepel_logits(ids):
    config, stored = decoder_config("kikepel-2048"), read_weights(weights_path("kikepel-2048") / "model.safetensors")
    eps, T = config["norm"]["eps"], len(ids)

    def w(name):
        return stored[name].double()

    def norm(x, name):
        return rms(x - x.mean(-1, keepdim=True), eps) * w(name)

    x = w("embed")[ids]
    for i, layer in enumerate(config["layers"]):
        m, p, f = layer["mixer"], f"l{i}.mix.", f"l{i}.mlp."
        H = m["heads"]
        q = (rms(x @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T
        c = rms(x @ w(p + "dkv").T, eps) * w(p + "dkv.norm")
        k, v = c @ w(p + "uk").T, c @ w(p + "uv").T
        o = softmax_attention(q.reshape(T, H, -1), k.reshape(T, H, -1), v.reshape(T, H, -1), m["scale"],
                              window=m["mask"]["size"], sink=w(p + "sink") if layer["type"] == "latent_attention" else None)
        x = x + norm(o.reshape(T, -1) @ w(p + "o").T, f"l{i}.norm1")
        if layer["mlp"]["kind"] == "dense":
            gate = torch.relu(x @ w(f + "gate").T + w(f + "gate.b"))
            y = (gate * (x @ w(f + "up").T + w(f + "up.b"))) @ w(f + "down").T + w(f + "down.b")
        else:
            y = mixture(x, w, f, layer["mlp"])
        x = x + norm(y, f"l{i}.norm2")
    cap = config["logit_softcap"]
    return cap * torch.tanh(norm(x, "final.norm") @ w("head").T * config["logit_scale"] / cap)


def exact(case, seed):
    ids = torch.from_numpy(token_ids(case, seed)).cuda()
    if case["model"] in HYENA:
        logits = hyena_logits(case["model"], ids)
    else:
        logits = gigusun_logits(ids) if case["model"] == "gigusun-2048" else kikepel_logits(ids)
    if case["kind"] != "generate":
        return logits
    return {"prompt": logits[:case["tokens"]], "steps": logits[case["tokens"]:]}
