"""GPU: the kernels of a prefill block and the batched routing of a decode step at the edges of their tiles."""
import pytest
import torch

from tests.helpers import SCENARIOS, TOL_BF16, orc, rel_err
from tests.scenarios import randomize_weights
from tests.test_parity_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Dh,H,Hkv,W,Me,Ms,norm", [(64, 4, 2, 50, 9, 5, "full"), (64, 3, 1, 64, 32, 32, "identity"),
                                                   (128, 2, 1, 40, 8, 16, "full"), (128, 8, 1, 100, 70, 22, "identity")])
@pytest.mark.parametrize("block,L", [(1, 3), (63, 130), (64, 192), (65, 131), (128, 320), (200, 333)])
def test_prefill_attention_at_tile_edges(Dh, H, Hkv, W, Me, Ms, norm, block, L):
    """64-row query tiles and 64-key tiles, their remainders, prefix tiles without a visible slot (fresh states: the first
    block reads none, later ones skip the banks that are still empty) against the shape-generic kernel (bf16; P and the two
    streams are rounded to bf16 at different places: a few 2^-9 of the result)."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, _deep_copy_state
    torch.manual_seed(3)
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=W, num_landmarks_exact=Me,
                               num_landmarks_summary=Ms, head_norm_mode=norm).eval()
    randomize_weights(mod, 3)
    mod = mod.to(torch.bfloat16).cuda()
    x = orc.mixture_inputs(3, L, H * Dh, centroids=16, sigma=0.3, seed=5, dtype=torch.bfloat16).cuda()
    sa = mod.init_state(batch_size=3, device="cuda", dtype=torch.bfloat16)
    sb = _deep_copy_state(sa)
    ya, sa = mod.prefill_chunked(x, sa, block_size=block)
    assert mod.device_status() == 0
    mod.use_tuned_kernels = False
    yb, sb = mod.prefill_chunked(x, sb, block_size=block)
    assert torch.equal(sa.k_buf, sb.k_buf) and torch.equal(sa.allowed, sb.allowed)
    assert rel_err(ya, yb) < 8e-3


@pytest.mark.parametrize("Dh", [64, 128])
def test_prefill_attention_weight_of_the_dominating_key_is_exact(Dh):
    """Two visible slots, one in each of the first two 64-key tiles, the second 2^6..2^8 times as heavy as the first, the same
    value behind every visible key: whatever the weights, the output is that value.  The heavy key's weight must be the 1 that
    bf16 holds exactly; taken against the first tile's maximum it is rounded by more than half a step of the value (keys
    chosen so), and the output is the next bf16 value."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    W, L, v = 128, 8, 1.9921875                              # v: half a bf16 step is 2^-8, 0.196 % of it
    s = torch.arange(0, 2000).mul(2.0 ** -5).to(torch.bfloat16).double().unique()     # candidate keys, query 8 in their place
    w = torch.exp(s * 8.0 / Dh ** 0.5)
    keep = (w > 2.0 ** 6) & (w < 2.0 ** 7.9) & ((w.float().to(torch.bfloat16).double() - w) / (w + 1) > 2.2e-3)
    s = s[keep]
    B = s.numel()
    assert B >= 3
    mod = CoDAGQALandmarkPerf2(embed_dim=2 * Dh, num_heads=2, num_kv_heads=1, window=W, num_landmarks_exact=0,
                               num_landmarks_summary=0, head_norm_mode="identity").eval().to(torch.bfloat16).cuda()
    st = mod.init_state(batch_size=B, device="cuda", dtype=torch.bfloat16)
    st.v_buf.fill_(v)
    for b in range(B):
        heavy = 64 + 7 * b % 64
        st.allowed[b, [5, heavy]] = True
        st.k_buf[b, 0, heavy, 0] = s[b].float()
    q, k, val = (torch.zeros(B, L, n * Dh, device="cuda", dtype=torch.bfloat16) for n in (2, 1, 1))
    q[..., 0] = q[..., Dh] = 8.0
    k[..., 0], val[:] = -100.0, v                            # the block's own keys weigh nothing
    lam, out = torch.zeros(B, L, 2, device="cuda"), torch.empty_like(q)
    mod._attend_block_tc(mod._cfg(B, torch.bfloat16, st), st, L, 0, L, q, q.clone(), lam, k, val, out)
    assert mod.device_status() == 0
    assert torch.equal(out, torch.full_like(out, v))


@pytest.mark.parametrize("Dh", [32, 64, 128])
@pytest.mark.parametrize("Lq,blk,Lbuf,used", [(1, False, 70, 0.5), (1, False, 200, 0.02), (2, True, 33, 0.0), (3, True, 40, 0.6),
                                              (8, True, 96, 1.0), (9, True, 31, 0.3), (65, True, 130, 0.1), (130, True, 5, 0.0),
                                              (1, False, 20, 0.5), (4, True, 12, 0.5), (5, True, 27, 0.9), (4, True, 60, 0.7), (4, True, 100, 0.4)])
def test_single_precision_attention(Dh, Lq, blk, Lbuf, used):
    """The register-tiled fp32 kernel (every row count per tile, keys split over one, two and four warps, tiles without a visible key)
    against the same attention in 64 bits; 32-bit sums over at most 260 keys."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    H, Hkv, B = 4, 2, 2
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=Lbuf, num_landmarks_exact=0,
                               num_landmarks_summary=0).eval().cuda()
    st = mod.init_state(batch_size=B, device="cuda", dtype=torch.float32)
    g = torch.Generator("cuda").manual_seed(Dh + Lq + Lbuf)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    st.k_buf.copy_(rnd(*st.k_buf.shape))
    st.v_buf.copy_(rnd(*st.v_buf.shape))
    st.allowed.copy_(torch.rand(B, Lbuf, generator=g, device="cuda") < used)
    q, qn = 2 * rnd(B, Lq, H * Dh), 2 * rnd(B, Lq, H * Dh)
    lam = torch.rand(B, Lq, H, generator=g, device="cuda")
    k, v = (rnd(B, Lq, Hkv * Dh), rnd(B, Lq, Hkv * Dh)) if blk else (None, None)
    with torch.no_grad():
        mod.head_norm.weight.copy_(rnd(Dh))
    out = torch.full((B, Lq, H * Dh), float("nan"), device="cuda")
    mod._attend(mod._cfg(B, torch.float32, st), st, Lq, q, qn, lam, k, v, out)

    d = lambda t: t.double()  # noqa: E731
    keys, vals = d(st.k_buf), d(st.v_buf)
    vis = st.allowed.bool()[:, None, :].expand(B, Lq, Lbuf)
    if blk:
        keys = torch.cat([keys, d(k).view(B, Lq, Hkv, Dh).transpose(1, 2)], 2)
        vals = torch.cat([vals, d(v).view(B, Lq, Hkv, Dh).transpose(1, 2)], 2)
        vis = torch.cat([vis, torch.ones(Lq, Lq, device="cuda").tril().bool().expand(B, Lq, Lq)], 2)
    keys, vals = (t.repeat_interleave(H // Hkv, 1) for t in (keys, vals))

    def stream(x):
        s = d(x).view(B, Lq, H, Dh).transpose(1, 2) @ keys.transpose(2, 3) / Dh ** 0.5
        return torch.softmax(s.masked_fill(~vis[:, None], float("-inf")), -1).nan_to_num(0.0) @ vals

    y = stream(q) - d(lam).transpose(1, 2)[..., None] * stream(qn)
    y = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + mod.eps) * d(mod.head_norm.weight)
    assert rel_err(out, y.transpose(1, 2).reshape(B, Lq, H * Dh)) < 5e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("Dh", [32, 64, 128])
def test_single_precision_attention_keeps_later_tokens_out(Dh, bad):
    """A token whose values are infinite or not a number leaves the outputs of the block's earlier tokens as they are, bit for
    bit, wherever it stands in the query and key tiles."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    mod = CoDAGQALandmarkPerf2(embed_dim=2 * Dh, num_heads=2, num_kv_heads=1, window=40, num_landmarks_exact=0,
                               num_landmarks_summary=0).eval().cuda()
    st = mod.init_state(batch_size=1, device="cuda", dtype=torch.float32)
    g = torch.Generator("cuda").manual_seed(Dh)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    st.k_buf.copy_(rnd(*st.k_buf.shape))
    st.v_buf.copy_(rnd(*st.v_buf.shape))
    st.allowed.fill_(True)
    cfg = mod._cfg(1, torch.float32, st)
    for Lq in (2, 3, 9, 40):
        q, qn, lam = rnd(1, Lq, 2 * Dh), rnd(1, Lq, 2 * Dh), torch.rand(1, Lq, 2, generator=g, device="cuda")
        k, v = rnd(1, Lq, Dh), rnd(1, Lq, Dh)
        want, out = torch.empty_like(q), torch.empty_like(q)
        mod._attend(cfg, st, Lq, q, qn, lam, k, v, want)
        for t in range(1, Lq):
            spoiled = v.clone()
            spoiled[0, t] = bad
            mod._attend(cfg, st, Lq, q, qn, lam, k, spoiled, out)
            assert torch.equal(out[:, :t], want[:, :t]), (Lq, t)
            assert not torch.isfinite(out[:, t:]).any()


@pytest.mark.parametrize("kw,Te,Ts,block,B", [
    # one warp per slot: more candidates than a warp has lanes, more than 16 LRU victims, slot counts that are not
    # multiples of 32, one and several tiles of scores
    (dict(num_heads=4, num_kv_heads=2, embed_dim=128, num_landmarks_exact=40, num_landmarks_summary=33), 40, 70, 96, 2),
    (dict(num_heads=3, num_kv_heads=3, embed_dim=192, num_landmarks_exact=70, num_landmarks_summary=100), 33, 90, 100, 2),
    (dict(num_heads=2, num_kv_heads=2, embed_dim=256, num_landmarks_exact=8, num_landmarks_summary=32), 8, 64, 48, 3),
    # rows above 256 elements: eight warps per slot; one KV head: no cluster
    (dict(num_heads=8, num_kv_heads=8, embed_dim=512, num_landmarks_exact=12, num_landmarks_summary=1), 5, 64, 70, 1),
    (dict(num_heads=2, num_kv_heads=1, embed_dim=128, num_landmarks_exact=1, num_landmarks_summary=3), 8, 64, 64, 2),
    # as many exact slots as the decisions' shared memory holds (33 bytes each were enough for 6000)
    (dict(num_heads=2, num_kv_heads=2, embed_dim=64, num_landmarks_exact=6000, num_landmarks_summary=4), 8, 64, 50, 1),
    # head_dim 20 and 12: chunks that straddle heads and the phase-safe half
    (dict(num_heads=4, num_kv_heads=2, embed_dim=80, num_landmarks_exact=16, num_landmarks_summary=16), 8, 64, 40, 2),
    (dict(num_heads=4, num_kv_heads=4, embed_dim=48, num_landmarks_exact=5, num_landmarks_summary=7), 3, 9, 33, 2),
])
def test_block_routing_matches_oracle(monkeypatch, kw, Te, Ts, block, B):
    """Scores, decisions, slot writes and events of the block write in fp32: occupancy, stamps and counters exactly, bank
    contents and outputs to the parity tolerance."""
    sc = dict(model=dict(window=32, exact_candidates_per_block=Te, summary_candidates_per_block=Ts, collect_metrics=True, **kw),
              model_seed=7, state_seed=9, B=B, random_gate=True,
              inputs=dict(kind="mixture", centroids=48, sigma=0.3, seed=11, L=4 * block + 40, Ldec=3),
              phases=[("prefill", 0, 4 * block + 40, block), ("decode", 0, 3)])
    monkeypatch.setitem(SCENARIOS, "block_routing", sc)
    _run("block_routing", check_golden=False)


@pytest.mark.parametrize("kw,B,narrow", [
    # 128-thread CTAs: more slots, stamps and cache chunks than threads, caches staged; the same unstaged (more than 30 KB); few of each
    (dict(embed_dim=256, num_heads=4, num_kv_heads=4, window=700, num_landmarks_exact=140, num_landmarks_summary=60), 100, True),
    (dict(embed_dim=256, num_heads=4, num_kv_heads=4, window=64, num_landmarks_exact=200, num_landmarks_summary=100), 100, True),
    (dict(embed_dim=192, num_heads=3, num_kv_heads=3, window=32, num_landmarks_exact=32, num_landmarks_summary=32), 150, True),
    # 256-thread CTAs: the same, and one KV head
    (dict(embed_dim=256, num_heads=4, num_kv_heads=4, window=700, num_landmarks_exact=140, num_landmarks_summary=60), 2, False),
    (dict(embed_dim=512, num_heads=8, num_kv_heads=1, window=33, num_landmarks_exact=5, num_landmarks_summary=90), 7, False),
    # the attention's lines between one and two CTAs per SM: two short tiles, six tiles below and above three planes per SM, one query head
    (dict(embed_dim=256, num_heads=4, num_kv_heads=1, window=100, num_landmarks_exact=12, num_landmarks_summary=12), 160, False),
    (dict(embed_dim=576, num_heads=9, num_kv_heads=3, window=300, num_landmarks_exact=40, num_landmarks_summary=40), 95, False),
    (dict(embed_dim=576, num_heads=9, num_kv_heads=3, window=300, num_landmarks_exact=40, num_landmarks_summary=40), 155, True),
    (dict(embed_dim=256, num_heads=4, num_kv_heads=4, window=300, num_landmarks_exact=40, num_landmarks_summary=40), 120, True),
])
def test_batched_routing_head_dim_64(kw, B, narrow):
    """The all-layers routing launch with 128 and with 256 threads per CTA and the token-writing attention with one and with two
    CTAs per SM, through the captured step against eager steps: the same bits in both banks."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chains = 2 * B * kw["num_kv_heads"]
    # 256-thread CTAs fit an SM four or five times, 128-thread ones at least 6.6 times: two rounds against one, or one round of either
    assert 5 * sms < chains <= 6.6 * sms if narrow else chains <= 4 * sms
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, CoDAStack, _deep_copy_state
    torch.manual_seed(5)
    layers = [CoDAGQALandmarkPerf2(**kw).eval() for _ in range(2)]
    for i, layer in enumerate(layers):
        randomize_weights(layer, 5 + i)
    layers = [layer.to(torch.bfloat16).cuda() for layer in layers]
    T, D = kw["window"] + 150, kw["embed_dim"]
    x = orc.mixture_inputs(B, T + 20, D, centroids=16, sigma=0.3, seed=8, dtype=torch.bfloat16).cuda()
    states = []
    for layer in layers:
        st = layer.init_state(batch_size=B, device="cuda", dtype=torch.bfloat16)
        layer.prefill_chunked(x[:, :T], st, block_size=64, return_outputs=False)
        states.append(st)
    twins = [_deep_copy_state(s) for s in states]
    stack = CoDAStack(layers)
    tok = x[:, T:T + 1].contiguous()
    stack.capture_step(states, tok)
    for t in range(T, T + 20):
        tok = x[:, t:t + 1].contiguous()
        y = stack.step_graph(tok, states)
        h = tok
        for layer, st in zip(layers, twins):
            o, _ = layer.step(h, st)
            h = h + o
        assert rel_err(y, h) < TOL_BF16
    # (the captured projections may round elsewhere, but every token evicted here was written by the shared prefill)
    W = kw["window"]
    for a, b in zip(states, twins):
        assert torch.equal(a.allowed, b.allowed) and torch.equal(a.mem_last_exact, b.mem_last_exact)
        assert torch.equal(a.k_buf[:, :, W:], b.k_buf[:, :, W:]) and torch.equal(a.v_buf[:, :, W:], b.v_buf[:, :, W:])
        assert torch.equal(a._exact_v_norm, b._exact_v_norm) and torch.equal(a._sum_lf_k_norm, b._sum_lf_k_norm)
    assert all(layer.device_status() == 0 for layer in layers)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("K,N,bias,res", [(512, 832, True, False), (4096, 4096, False, True), (1024, 6208, True, True)])
def test_skinny_gemm_row_instances(M, K, N, bias, res):
    """Every number of 8-row tiles of the four-way kernel against the product in 64 bits: fp32 sums, one rounding of the product
    and one of the sum with the residual (2^-8 of a value together, in the norm well below)."""
    from coda_gqa_l_b200 import _lib as b
    g = torch.Generator("cuda").manual_seed(M + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, w = rnd(M, K), rnd(N, K)
    bv, rv = (rnd(N) if bias else None), (rnd(M, N) if res else None)
    y = torch.full((M + 1, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    b.check(b.lib.coda_b200_skinny_gemm_bias(x.data_ptr(), M, K, w.data_ptr(), N, p(bv), p(rv), N, y.data_ptr(), N, status.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream), "skinny")
    want = x.double() @ w.double().t()
    if bias:
        want = want + bv.double()
    if res:
        want = want + rv.double()
    assert status.item() == 0 and torch.isnan(y[M]).all()
    assert rel_err(y[:M], want) < 4e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hkv,Dh,Me,Ms", [(4, 2, 64, 7, 5), (2, 1, 20, 1, 0), (8, 8, 128, 0, 33), (2, 2, 64, 0, 0)])
def test_routing_caches_of_a_fresh_state(dtype, H, Hkv, Dh, Me, Ms):
    """The one-launch unit vectors against torch's normalisation of the same slots, zeros for zero rows.  The norm's 32-bit sum
    runs in another order: at most 7 roundings each way, halved by the root, and one of the quotient, below 2^-21; in bf16 a
    norm or a quotient that falls on the other side moves by one step, at most 2^-7."""
    from torch.nn import functional as F
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=6, num_landmarks_exact=Me,
                               num_landmarks_summary=Ms).eval().to(dtype).cuda()
    ulp = 2.0 ** -21 if dtype == torch.float32 else 2.0 ** -7
    for init in ("random_normal", "zeros"):
        st = mod.init_state(batch_size=3, device="cuda", dtype=dtype, mem_init=init)
        for got, src in ((st._exact_v_norm, st.v_buf[:, :, 6:6 + Me]), (st._sum_lf_k_norm, st.k_buf[:, :, 6 + Me:, Dh // 2:])):
            if got is not None:
                assert torch.allclose(got.double(), F.normalize(src, dim=-1, eps=1e-6).double(), rtol=ulp, atol=0)



@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("interleaved,Dh,H,Hkv", [(True, 128, 3, 1), (False, 64, 3, 3), (True, 24, 2, 1), (False, 32, 4, 2)])
@pytest.mark.parametrize("B,L", [(2, 1), (1, 1184), (70, 37), (331, 37), (5, 1201)])
def test_projection_postprocessing_tiles(dtype, interleaved, Dh, H, Hkv, B, L):
    """The vector kernel's tiles of one token, of several positions, of positions and states, and their remainders, against the
    element-wise kernel (rows that start one element off a 16-byte boundary): the same operations, so the same bits."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    torch.manual_seed(1)
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=16, num_landmarks_exact=4,
                               num_landmarks_summary=4, rope_interleaved=interleaved, rope_base=1e6).eval()
    randomize_weights(mod, 2)
    mod = mod.to(dtype).cuda()
    cfg = mod._cfg(B, dtype, mod.init_state(batch_size=B, device="cuda", dtype=dtype))
    nq, nk = H * Dh, Hkv * Dh
    n = nq + nk + H + 1
    src = torch.randn(B, L, n, generator=torch.Generator("cuda").manual_seed(4), device="cuda").to(dtype)
    outs = []
    for shift in (0, 1):
        y = torch.zeros(B, L, (n + 16) // 8 * 8, device="cuda", dtype=dtype)
        y[..., shift:shift + n] = src
        q, k, lam_logit, gate_logit = y[..., shift:shift + n].split([nq, nk, H, 1], -1)
        qn, lam, gate = mod._prep(cfg, L, 1000, q, k, lam_logit, gate_logit, True)
        outs.append((q, k, qn, lam, gate))
    for a, b, name in zip(*outs, ("q", "k", "q_noise", "lambda", "gate")):
        assert torch.equal(a, b), name
    assert not torch.equal(outs[0][0], src[..., :nq]) and not torch.equal(outs[0][0], outs[0][2])


def test_step_whose_output_projection_is_refused_keeps_its_token():
    """The one-call step writes the cache before the output projection: where that is refused (here by a width the GEMM does not
    take, on the host), the error is raised and the ring scalars tell that the token is in, as when the calls were separate."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, _deep_copy_state
    torch.manual_seed(2)
    mod = CoDAGQALandmarkPerf2(embed_dim=256, num_heads=4, num_kv_heads=2, window=6, num_landmarks_exact=4,
                               num_landmarks_summary=4).eval().to(torch.bfloat16).cuda()
    x = torch.randn(12, 2, 1, 256, device="cuda", dtype=torch.bfloat16)
    st = mod.init_state(batch_size=2, device="cuda", dtype=torch.bfloat16)
    for t in range(10):
        mod.step(x[t], st)
    twin = _deep_copy_state(st)
    mod.step(x[10], twin)
    bd = mod._decode_bundle(x.device, x.dtype)
    assert mod._one_call_ok(bd, 2)
    bd["layer"].n_out = 100
    with pytest.raises(RuntimeError, match="skinny_gemm"):
        mod.step(x[10], st)
    bd["layer"].n_out = bd["n_out"]
    assert (st.pos, st.recent_idx, st.recent_filled) == (twin.pos, twin.recent_idx, twin.recent_filled)
    ya, yb = mod.step(x[11], st)[0], mod.step(x[11], twin)[0]
    assert torch.equal(ya, yb) and torch.equal(st.k_buf, twin.k_buf) and torch.equal(st.v_buf, twin.v_buf)


def test_quotients_of_bf16_values_are_the_divisions():
    """The device's bf16 quotient from an approximate reciprocal, seen through the unit vectors of a fresh state's slots: a row
    holds one value b and values 2^-12 as large, so that its norm rounds to b exactly; every pair of significands, both signs,
    with b from 2^-12 to 2^60, and rows below the smallest denominator (1e-6), down to subnormal values; equal bits."""
    import ctypes as C
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, _lib as lib
    Dh, Me = 128, 256
    mod = CoDAGQALandmarkPerf2(embed_dim=Dh, num_heads=1, num_kv_heads=1, window=4, num_landmarks_exact=Me,
                               num_landmarks_summary=0).eval().to(torch.bfloat16).cuda()
    scales = [0, -12, 20, 60, -22, -60, -100, -118]
    st = mod.init_state(batch_size=len(scales), device="cuda", dtype=torch.bfloat16, mem_init="zeros")
    sig = 1.0 + torch.arange(128, device="cuda", dtype=torch.float64) / 128
    rows = torch.empty(Me, Dh, device="cuda", dtype=torch.float64)     # row 2 i + j: b = sig[i], the others sig[j:j + 127]
    rows[:, 0] = sig.repeat_interleave(2)
    for j in range(2):
        rows[j::2, 1:] = sig[j:j + 127] * 2.0 ** -12 * torch.tensor([1.0, -1.0], device="cuda").repeat(64)[:127]
    for b, e in enumerate(scales):
        st.v_buf[b, 0, 4:] = (rows * 2.0 ** e).to(torch.bfloat16)
    x = st.v_buf[:, 0, 4:].clone()
    ptrs = mod._ptrs(st)
    lib.check(lib.lib.coda_b200_bank_norms(C.byref(mod._cfg(len(scales), torch.bfloat16, st)), C.byref(ptrs),
                                           torch.cuda.current_stream().cuda_stream), "bank_norms")
    smallest = torch.tensor(1e-6).to(torch.bfloat16).float().cuda()
    for b, e in enumerate(scales):
        den = torch.maximum(x[b, :, :1].float(), smallest)
        assert torch.equal(st._exact_v_norm[b, 0], (x[b].float() / den).to(torch.bfloat16)), e


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("Lbuf,blk,scale", [(130, 64, 2.0), (384, 256, 0.5), (200, 333, 2.0), (768, 65, 6.0), (70, 1, 2.0)])
def test_prefill_attention_error_against_64_bits(Dh, Lbuf, blk, scale):
    """bf16 weights and a bf16 result, everything else in 32 bits: each weight off by at most 2^-8 of itself (and 1e-4 where its
    exponential is a polynomial; 2^-16 for 32-bit sums), the result rounded once.  Bound per element, from the absolute values."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2
    H, Hkv, B = 4, 2, 2
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=Lbuf, num_landmarks_exact=0,
                               num_landmarks_summary=0, head_norm_mode="identity").eval().to(torch.bfloat16).cuda()
    st = mod.init_state(batch_size=B, device="cuda", dtype=torch.bfloat16)
    g = torch.Generator("cuda").manual_seed(Dh + Lbuf + blk)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    st.k_buf.copy_(rnd(*st.k_buf.shape))
    st.v_buf.copy_(rnd(*st.v_buf.shape))
    st.allowed.copy_(torch.rand(B, Lbuf, generator=g, device="cuda") < 0.8)
    q, qn, k, v = scale * rnd(B, blk, H * Dh), scale * rnd(B, blk, H * Dh), rnd(B, blk, Hkv * Dh), rnd(B, blk, Hkv * Dh)
    lam = torch.rand(B, blk, H, generator=g, device="cuda").to(torch.bfloat16).float()
    out = torch.full((B, blk, H * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    mod._attend_block_tc(mod._cfg(B, torch.bfloat16, st), st, blk, 0, blk, q, qn, lam, k, v, out)
    assert mod.device_status() == 0

    heads = lambda t, n: t.double().view(B, blk, n, Dh).transpose(1, 2)  # noqa: E731
    keys = torch.cat([st.k_buf.double(), heads(k, Hkv)], 2).repeat_interleave(H // Hkv, 1)
    vals = torch.cat([st.v_buf.double(), heads(v, Hkv)], 2).repeat_interleave(H // Hkv, 1)
    vis = torch.cat([st.allowed.bool()[:, None].expand(B, blk, Lbuf),
                     torch.ones(blk, blk, device="cuda").tril().bool().expand(B, blk, blk)], 2)[:, None]
    w = [torch.softmax((heads(x, H) @ keys.transpose(2, 3) / Dh ** 0.5).masked_fill(~vis, float("-inf")), -1) for x in (q, qn)]
    lam = lam.double().transpose(1, 2)[..., None]
    want = w[0] @ vals - lam * (w[1] @ vals)
    bound = (2.0 ** -8 + 1e-4 + 2.0 ** -16) * (w[0] @ vals.abs() + lam * (w[1] @ vals.abs())) + 2.0 ** -8 * want.abs()
    err = (heads(out, H) - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("Dh,dtype", [(64, torch.bfloat16), (128, torch.bfloat16), (64, torch.float32), (20, torch.bfloat16)])
def test_prefill_replayed_from_a_graph(Dh, dtype):
    """The chained launches of a prefill's blocks captured and replayed: the bits of the plain call in the output and the state."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, _deep_copy_state
    torch.manual_seed(5)
    mod = CoDAGQALandmarkPerf2(embed_dim=4 * Dh, num_heads=4, num_kv_heads=2, window=96, num_landmarks_exact=16,
                               num_landmarks_summary=16).eval()
    randomize_weights(mod, 3)
    mod = mod.to(dtype).cuda()
    x = orc.mixture_inputs(3, 400, 4 * Dh, centroids=16, sigma=0.3, seed=5, dtype=dtype).cuda()
    st = mod.init_state(batch_size=3, device="cuda", dtype=dtype)
    mod.prefill_chunked(x[:, :200].contiguous(), st, block_size=64)
    rest = x[:, 200:].contiguous()
    twin, warm = _deep_copy_state(st), _deep_copy_state(st)
    want, twin = mod.prefill_chunked(rest, twin, block_size=64)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        mod.prefill_chunked(rest, warm, block_size=64)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y, st = mod.prefill_chunked(rest, st, block_size=64)
    graph.replay()
    assert torch.equal(y, want) and (st.pos, st.recent_idx, st.recent_filled) == (twin.pos, twin.recent_idx, twin.recent_filled)
    for f in ("k_buf", "v_buf", "allowed", "g_recent", "mem_last_exact", "_exact_v_norm", "_sum_lf_k_norm"):
        assert torch.equal(getattr(st, f), getattr(twin, f)), f
    assert mod.device_status() == 0
