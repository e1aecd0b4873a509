"""CPU: the selection-order routines compiled into the library (the same header the device kernels use)
return exactly the index lists of torch.topk on the host, ties included."""
import ctypes as C

import numpy as np
import pytest
import torch


def _lib():
    from coda_gqa_l_b200 import _lib
    return _lib.lib


def _topk(v: torch.Tensor, k: int, largest: bool, sorted_: bool):
    out = np.zeros(max(k, 1), dtype=np.int32)
    if v.dtype == torch.float32:
        a = np.ascontiguousarray(v.numpy(), dtype=np.float32)
        rc = _lib().coda_b200_host_topk_f32(a.ctypes.data, v.numel(), k, int(largest), int(sorted_), out.ctypes.data)
    else:
        a = np.ascontiguousarray(v.numpy(), dtype=np.int64)
        rc = _lib().coda_b200_host_topk_i64(a.ctypes.data, v.numel(), k, int(largest), int(sorted_), out.ctypes.data)
    assert rc == 0
    return out[:k].tolist()


def _gates(mode: int, n: int, g: torch.Generator) -> torch.Tensor:
    if mode == 0:
        return torch.full((n,), 0.11920292)                        # default constant gate
    if mode == 1:
        return torch.rand(n, generator=g)
    if mode == 2:
        return torch.randint(0, 3, (n,), generator=g).float()      # heavy ties
    v = torch.rand(n, generator=g)
    v[torch.rand(n, generator=g) < 0.5] = 0.5
    return v


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 31, 64, 65, 127, 128, 192, 256, 257, 512, 1000, 1024, 4096])
def test_gate_selection_order(n):
    g = torch.Generator().manual_seed(n)
    for k in (1, 2, 7, 8, 9, 16, 17, 33, 63, 64, 65):
        if k > n:
            continue
        for mode in range(4):
            v = _gates(mode, n, g)
            for largest, sorted_ in ((True, False), (True, True), (False, False), (False, True)):
                ref = torch.topk(v.view(1, n), k, dim=1, largest=largest, sorted=sorted_)[1][0].tolist()
                assert _topk(v, k, largest, sorted_) == ref, (n, k, mode, largest, sorted_)


@pytest.mark.parametrize("Me", [4, 8, 16, 32, 64, 128, 256])
def test_lru_victim_order(Me):
    g = torch.Generator().manual_seed(Me)
    for k in (1, 2, 4, 8, 16, 18, 32):
        if k > Me:
            continue
        for mode in range(3):
            for _ in range(4):
                if mode == 0:
                    v = torch.full((Me,), -(2 ** 62), dtype=torch.int64)
                else:
                    v = torch.randint(0, 1000, (Me,), generator=g)
                    if mode == 2:
                        v[torch.rand(Me, generator=g) < 0.4] = -(2 ** 62)
                ref = torch.topk(v.view(1, Me), k, dim=1, largest=False, sorted=True)[1][0].tolist()
                assert _topk(v, k, False, True) == ref, (Me, k, mode)


def test_known_answers():
    """Index lists measured on the host top-k for the shapes the default configurations hit."""
    const = lambda n: torch.full((n,), 0.11920292)  # noqa: E731
    assert _topk(const(256), 64, True, False)[:9] == [160, 191, 190, 189, 188, 187, 186, 185, 184]
    assert _topk(const(256), 8, True, False) == [172, 169, 170, 171, 174, 175, 168, 173]
    assert _topk(const(128), 64, True, False)[:4] == [96, 65, 66, 67]
    unused = lambda n: torch.full((n,), -(2 ** 62), dtype=torch.int64)  # noqa: E731
    assert _topk(unused(64), 8, False, True) == [44, 41, 42, 43, 46, 47, 40, 45]
    assert _topk(unused(32), 8, False, True) == [20, 23, 22, 21, 18, 17, 24, 19]


@pytest.mark.gpu
@pytest.mark.parametrize("W,fill0,L,block,Te,Ts", [
    (256, 256, 1024, 256, 8, 64), (256, 0, 1000, 1024, 8, 64), (128, 100, 517, 97, 8, 64), (64, 64, 640, 64, 3, 2),
    (16, 16, 4000, 4000, 8, 64), (32, 32, 6400, 6400, 8, 16), (8, 8, 48, 3, 8, 64), (64, 64, 192, 33, 33, 33)])
def test_device_selection_equals_host_topk(W, fill0, L, block, Te, Ts):
    """The warp's replay of the selection (partition passes by ballots and prefix counts) leaves the index lists of
    torch.topk on the host, in their order, for distinct, tied and mixed gates; exact: indices."""
    from coda_gqa_l_b200 import _lib as b
    B, nblk = 8, (L + block - 1) // block
    g = torch.Generator().manual_seed(W + L)
    gates = torch.stack([_gates(i % 4, fill0 + L, g) for i in range(B)])
    cfg = b.LayerCfg(B=B, H=2, Hkv=1, Dh=64, W=W, Me=4, Ms=4, dtype=b.CODA_F32, Te=Te, Ts=Ts)
    dev = gates.cuda()
    tmax = max(1, min(max(Te, Ts), block))
    cand = torch.full((B, nblk, tmax), -1, dtype=torch.int32, device="cuda")
    b.check(b.lib.coda_b200_select_candidates(C.byref(cfg), dev.data_ptr(), dev.stride(0), fill0, L, block, cand.data_ptr(), tmax,
                                              torch.cuda.current_stream().cuda_stream), "select")
    cand = cand.cpu()
    for j in range(nblk):
        seen = fill0 + j * block
        fill, blk = min(seen, W), min(block, L - j * block)
        n_ev = max(0, fill + blk - W)
        k = max(min(Te, n_ev), min(Ts, n_ev))
        if k == 0:
            continue
        for s in range(B):
            ref = torch.topk(gates[s:s + 1, seen - fill:seen - fill + n_ev], k, dim=1, sorted=False)[1][0].tolist()
            assert cand[s, j, :k].tolist() == ref, (s, j)
