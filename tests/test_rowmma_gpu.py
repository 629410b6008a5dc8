"""The batched GEMM of Q5_K, Q6_K and Q8_0 (csrc/kdnn_rowmma.cuh) at the edges of its tiles, against float64.

Bound: the integer sums are exact and each of a row's K / 16 partial products meets a handful of fp32 roundings, at most
K / 16 + 8 of them in a chain: |error| <= (K / 16 + 16) * 2^-23 * sum_k |W[j, k]| |q d|, min term included."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one 16-row tile and one past it, 32-row tiles; 8, 16 and 32 activation rows, one past each; fewer super-blocks than
# warps, as many, one more; odd super-block counts put Q6_K rows on every even offset
@pytest.mark.parametrize("N,K,M", [(1, 256, 4), (17, 512, 8), (33, 2048, 9), (130, 2304, 16), (63, 768, 17), (64, 1280, 33),
                                   (2400, 768, 5), (2399, 256, 16), (300, 1792, 70)])
@pytest.mark.parametrize("fmt", [O.Q5_K, O.Q6_K, O.Q8_0])
def test_gemm_edges(kd, fmt, N, K, M):
    w = kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(fmt, N, K, N + M, scale_bits=0x1C00), fmt, N, K, DEV)
    g = torch.Generator().manual_seed(M)
    X = torch.randn(M, K, generator=g)
    X[:, ::40] *= 30.0
    X[M // 2, :] = 0.0
    dense = torch.empty((N, K), dtype=torch.float32, device=DEV)
    kd.dequant_to_dense(w, dense)
    W = dense.cpu().numpy().astype(np.float64)
    b = X.numpy().reshape(M, -1, 32)
    amax = np.abs(b).max(-1, keepdims=True)
    inv = np.divide(np.float32(127.0), amax, out=np.zeros_like(amax), where=amax > 0)
    q = (np.clip(np.rint(b * inv), -127, 127).astype(np.float64) * (amax / np.float32(127.0)).astype(np.float64)).reshape(M, K)
    # a Q5_K weight is the difference of two larger numbers: eight times the block's largest weight covers both
    mag = np.abs(W).reshape(N, -1, 32).max(-1).repeat(32, 1) * (8 if fmt == O.Q5_K else 1)
    bound = (K / 16 + 16) * 2.0 ** -23 * (np.abs(q) @ mag.T)
    out = {}
    for dtype in (torch.float32, torch.bfloat16):
        Y = torch.full((M + 1, N), float("nan"), dtype=dtype, device=DEV)
        ws = torch.zeros(kd.quant_gemm_workspace_bytes(M, K), dtype=torch.uint8, device=DEV)
        kd.quant_gemm(X.to(DEV), w, Y[:M], ws)
        torch.cuda.synchronize()
        assert bool(torch.isnan(Y[M]).all())
        out[dtype] = Y[:M]
    assert np.all(np.abs(out[torch.float32].cpu().numpy().astype(np.float64) - q @ W.T) <= bound)
    assert torch.equal(out[torch.bfloat16], out[torch.float32].to(torch.bfloat16))
