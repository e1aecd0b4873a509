"""What the bounded-cache attention path is timed on: decode steps and prefills as user programs run them.

A case is a dict of plain values.  ``kind`` says which public entry point a pass goes through:

* ``step``     one token through one layer's ``step`` (eager launches)
* ``adapter``  one token through a chain of ``LlamaCoDAAdapter`` modules, the residual added by the host program
* ``graph``    one token for every state through ``CoDAStack.step_graph`` (inputs on the device)
* ``host``     the same through ``CoDAStack.step_graph_host`` (pinned host token in, host result out)
* ``prefill``  the next ``L`` tokens of every state through ``prefill_chunked``, on states that have tokens behind them
* ``prompt``   a new prompt of ``L`` tokens through a ``LlamaCoDAAdapter`` with no state yet: it makes one, then prefills

The layer shapes are those of this repository's benchmark and tests (``SHAPES``).  Weights are the modules' seeded
default initialisation with the learned scalars moved off their constants, hidden states come from a seeded Gaussian
mixture.  Every pass returns the output and the whole updated state of every layer it ran.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "coda-gqa-l_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, CoDAStack, LlamaCoDAAdapter  # noqa: E402

# embed, query heads, KV heads, ring window, exact slots, summary slots, RoPE base, head norm, interleaved pairs,
# centroids and spread of the hidden-state mixture
SHAPES = {
    "d512": dict(D=512, H=8, Hkv=2, W=256, Me=64, Ms=64, base=1e4, norm="full", inter=True, K=512, sigma=0.3),
    "d576": dict(D=576, H=9, Hkv=3, W=128, Me=32, Ms=32, base=1e4, norm="identity", inter=False, K=1024, sigma=0.3),
    "d4096": dict(D=4096, H=32, Hkv=8, W=256, Me=64, Ms=64, base=1e6, norm="identity", inter=False, K=4096, sigma=0.5),
    "d8192": dict(D=8192, H=64, Hkv=8, W=512, Me=128, Ms=128, base=1e6, norm="identity", inter=False, K=8192, sigma=0.5),
}
TAPE = 16           # decode tokens per state that a prepared case walks through


def listed():
    def decode(name, kind, shape, B, layers, dtype="bf16"):
        return dict(name=name, kind=kind, shape=shape, B=B, layers=layers, dtype=dtype)

    def prefill(name, kind, shape, B, L, block, dtype="bf16"):
        return dict(name=name, kind=kind, shape=shape, B=B, L=L, block=block, dtype=dtype)

    return [
        # the smallest call: one sequence, one small layer, token by token
        decode("step_d512_b1", "step", "d512", 1, 1),
        # one chat sequence in a model whose attention modules were swapped for adapters (four of its layers)
        decode("adapter_d4096_b1", "adapter", "d4096", 1, 4),
        # a serving batch at the 7B shape, 32 states per GPU (eight of its layers; weights and states exceed L2)
        decode("graph_d4096_b32", "graph", "d4096", 32, 8),
        # a fuller batch of odd size at the same shape
        decode("graph_d4096_b100", "graph", "d4096", 100, 4),
        # many states of a tiny model: small planes, small projections
        decode("graph_d576_b512", "graph", "d576", 512, 8),
        # the 70B shape fed from and answered to the host (three of its layers)
        decode("host_d8192_b64", "host", "d8192", 64, 3),
        # single precision, one sequence: the configuration parity is judged in
        prefill("prefill_d512_f32_b1", "prefill", "d512", 1, 2048, 256, "f32"),
        # a long stream for a batch of small layers
        prefill("prefill_d512_b64", "prefill", "d512", 64, 2048, 256),
        # a tiny model's prefill with many states
        prefill("prefill_d576_b512", "prefill", "d576", 512, 256, 128),
        # the 7B shape: one 512-token chunk for 32 states
        prefill("prefill_d4096_b32", "prefill", "d4096", 32, 512, 128),
        # the 70B shape: a 1024-token chunk for a few states
        prefill("prefill_d8192_b8", "prefill", "d8192", 8, 1024, 256),
        # a single user's prompt of ragged length arriving at an adapter with its default block size
        prefill("prompt_d4096_l1000", "prompt", "d4096", 1, 1000, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "adapter", "graph", "graph", "host", "prefill", "prefill", "prefill", "prompt"])
    if kind in ("step", "adapter"):
        shape = rng.choice(["d512", "d576", "d4096"] if kind == "step" else ["d4096", "d8192"])
        layers = 1 if kind == "step" else rng.randint(1, 4 if shape == "d4096" else 2)
        # single precision is a parity mode of the small layers
        dtype = "f32" if shape in ("d512", "d576") and rng.random() < 0.25 else "bf16"
        return dict(kind=kind, shape=shape, B=_log_int(rng, 1, 48), layers=layers, dtype=dtype)
    if kind in ("graph", "host"):
        shape = rng.choice(["d512", "d576", "d4096", "d8192"])
        most = {"d512": 256, "d576": 512, "d4096": 128, "d8192": 64}[shape]
        return dict(kind=kind, shape=shape, B=_log_int(rng, 1, most), dtype="bf16",
                    layers=rng.randint(1, {"d512": 8, "d576": 8, "d4096": 5, "d8192": 3}[shape]))
    if kind == "prompt":
        return dict(kind=kind, shape=rng.choice(["d576", "d4096"]), B=rng.randint(1, 4), L=_log_int(rng, 20, 2000),
                    block=1024, dtype="bf16")
    shape = rng.choice(["d512", "d576", "d4096", "d8192"])
    dtype = "f32" if shape in ("d512", "d576") and rng.random() < 0.25 else "bf16"
    most = {"d512": 131072, "d576": 131072, "d4096": 16384, "d8192": 8192}[shape] // (8 if dtype == "f32" else 1)
    L = _log_int(rng, 32, 4096)
    return dict(kind=kind, shape=shape, B=_log_int(rng, 1, max(1, min(512, most // L))), L=L,
                block=rng.choice([64, 128, 256, 512]), dtype=dtype)


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _mixture(s, B, L, gen, dtype):
    cent = torch.randn(s["K"], s["D"], generator=gen, device="cuda")
    ids = torch.randint(0, s["K"], (B, L), generator=gen, device="cuda")
    x = torch.empty((B, L, s["D"]), device="cuda", dtype=dtype)
    step = max(1, (1 << 22) // (B * s["D"]))                 # (a few rows at a time: no fp32 copy of the whole input)
    for t in range(0, L, step):
        part = ids[:, t:t + step]
        x[:, t:t + step] = cent[part] + s["sigma"] * torch.randn((*part.shape, s["D"]), generator=gen, device="cuda")
    return x


def _seasoned(layer, gen):
    """Learned parameters away from the constants they start at: rotations, lambda, write gates and EMA rates differ."""
    def noise(t):
        return torch.randn(t.shape, generator=gen, device="cuda").to(t.dtype)
    with torch.no_grad():
        layer.theta.add_(0.3 * noise(layer.theta))
        layer.lambda_proj.bias.fill_(-1.0)
        layer.write_proj.weight.copy_(noise(layer.write_proj.weight) / math.sqrt(layer.embed_dim))
        layer.summary_eta_logit.add_(0.3 * noise(layer.summary_eta_logit))
    return layer


def _layer(s, dtype, gen):
    with torch.device("cuda"):
        layer = CoDAGQALandmarkPerf2(embed_dim=s["D"], num_heads=s["H"], num_kv_heads=s["Hkv"], window=s["W"],
                                     num_landmarks_exact=s["Me"], num_landmarks_summary=s["Ms"], rope_base=s["base"],
                                     head_norm_mode=s["norm"], rope_interleaved=s["inter"])
    return _seasoned(layer, gen).eval().to(dtype)


def _adapter(s, block, dtype, gen):
    with torch.device("cuda"):
        ad = LlamaCoDAAdapter(s["D"], s["H"], s["Hkv"], s["D"] // s["H"], bounded=True, rope_theta=s["base"],
                              window=s["W"], num_landmarks_exact=s["Me"], num_landmarks_summary=s["Ms"], block_size=block)
    _seasoned(ad.coda, gen)
    return ad.eval().to(dtype)


def _season_state(layer, state, s, B, gen, dtype):
    """Tokens behind a state: its ring is full and tokens have been routed into both banks."""
    x = _mixture(s, B, s["W"] + 2 * 128, gen, dtype)
    layer.prefill_chunked(x, state, block_size=128, return_outputs=False)


def prepare(case, seed):
    s, B, dtype = SHAPES[case["shape"]], case["B"], _dtype(case)
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"case": case, "i": 0}
    kind = case["kind"]
    if kind == "prompt":
        st["adapters"] = [_adapter(s, case["block"], dtype, gen)]
        st["x"] = _mixture(s, B, case["L"], gen, dtype)
        return st
    if kind == "prefill":
        st["layer"] = _layer(s, dtype, gen)
        st["states"] = [st["layer"].init_state(batch_size=B, device="cuda", dtype=dtype)]
        _season_state(st["layer"], st["states"][0], s, B, gen, dtype)
        st["x"] = _mixture(s, B, case["L"], gen, dtype)
        return st
    tokens = _mixture(s, B, TAPE, gen, dtype)
    st["tape"] = [tokens[:, t:t + 1].contiguous() for t in range(TAPE)]
    if kind == "adapter":
        st["adapters"] = [_adapter(s, 1024, dtype, gen) for _ in range(case["layers"])]
        for ad in st["adapters"]:
            _season_state(ad.coda, ad.init_inference_state(B, "cuda", dtype), s, B, gen, dtype)
        return st
    layers = [_layer(s, dtype, gen) for _ in range(case["layers"])]
    st["states"] = [layer.init_state(batch_size=B, device="cuda", dtype=dtype) for layer in layers]
    for layer, state in zip(layers, st["states"]):
        _season_state(layer, state, s, B, gen, dtype)
    if kind == "step":
        st["layer"] = layers[0]
        return st
    st["stack"] = CoDAStack(layers)
    if kind == "host":
        st["tape"] = [t.cpu().pin_memory() for t in st["tape"]]
    st["stack"].capture_step(st["states"], st["tape"][0])     # a serving program captures before it takes requests
    return st


def _state_tensors(state):
    return [state.k_buf, state.v_buf, state.allowed, state.g_recent, state.mem_last_exact,
            state._exact_v_norm, state._sum_lf_k_norm]


def run(st):
    kind = st["case"]["kind"]
    if kind == "prompt":
        ad, = st["adapters"]
        ad.reset_state()
        y = ad(st["x"])[0]
        return [y, _state_tensors(ad.get_state())]
    if kind == "prefill":
        y, st["states"][0] = st["layer"].prefill_chunked(st["x"], st["states"][0], block_size=st["case"]["block"])
        return [y, _state_tensors(st["states"][0])]
    x = st["tape"][st["i"] % TAPE]
    st["i"] += 1
    if kind == "step":
        y, st["states"][0] = st["layer"].step(x, st["states"][0])
        return [y, _state_tensors(st["states"][0])]
    if kind == "adapter":
        for ad in st["adapters"]:
            x = x + ad(x)[0]
        return [x] + [_state_tensors(ad.get_state()) for ad in st["adapters"]]
    if kind == "graph":
        y = st["stack"].step_graph(x, st["states"])
    else:
        y = st["stack"].step_graph_host(x, st["states"])
        torch.cuda.current_stream().synchronize()             # the host reads the result before it sends the next token
    return [y] + [_state_tensors(state) for state in st["states"]]


def work(case):
    s, B, e = SHAPES[case["shape"]], case["B"], 4 if case["dtype"] == "f32" else 2
    D, H, Hkv, W, Me, Ms = s["D"], s["H"], s["Hkv"], s["W"], s["Me"], s["Ms"]
    Dh, Lbuf = D // H, W + Me + Ms
    params = D * (H * Dh + 2 * Hkv * Dh + H + 1) + H * Dh * D
    caches = Hkv * (Me * Dh + Ms * (Dh // 2)) * e                           # routing caches of one state
    row = 2 * Hkv * Dh * e                                                  # one K/V slot of one state
    if "L" not in case:
        # per layer: weights, every slot, the routing caches, one written ring, exact and summary slot
        per = params * e + B * (row * Lbuf + caches + 3 * row + Lbuf)
        flops = B * (2.0 * params + 8.0 * H * Dh * Lbuf)
        return {"bytes": float(case["layers"] * per + 2 * B * D * e), "flops": case["layers"] * flops}
    L, blk = case["L"], case["block"]
    fresh = case["kind"] == "prompt"
    keys, t = 0.0, 0                                                        # visible keys summed over the queries
    while t < L:
        n = min(blk, L - t)
        prefix = Lbuf if not fresh else min(t, Lbuf)
        keys += n * (prefix + (n + 1) / 2)
        t += n
    state = B * (row * Lbuf + caches)
    bytes_ = params * e + 2 * B * L * D * e + (0 if fresh else state) + B * row * min(L, W) + B * caches
    return {"bytes": float(bytes_), "flops": B * (2.0 * L * params + 8.0 * H * Dh * keys)}


def tolerance(case):
    # Measured over the listed and some drawn cases, the tuned against the shape-generic kernels (other summation orders,
    # P rounded to bf16 at another place): bf16 up to 7e-3 in the norm (seven layers; one layer 5e-3) and 0.065 of the
    # rms in one value, no whole value differing.  Single precision: 32-bit sums over at most 4096 terms.
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.0}
    return {"rel": 2e-2, "max": 0.25, "differ": 1e-3}
