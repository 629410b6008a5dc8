"""The split-fp16 tensor-core kernel (csrc/kdnn_split.cuh) at the edges of its tiles, against float64.

Bound: an activation is represented to 2^-23 of its 256-element group's largest value, everything else is fp32
rounding of sums of at most K terms: |error| <= 2^-19 * max|W row| * sum_k (group maximum of |x|)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _exact(kd, w, X):
    """(float64 product with the int8-quantized rows, bound) -- weights from the bit-exact dequantizer."""
    dense = torch.empty((w.rows, w.cols), dtype=torch.float32, device=DEV)
    kd.dequant_to_dense(w, dense)
    b = X.float().cpu().numpy().reshape(X.shape[0], -1, 32)
    amax = np.abs(b).max(-1, keepdims=True)
    inv = np.divide(np.float32(127.0), amax, out=np.zeros_like(amax), where=amax > 0)
    q = np.clip(np.rint(b * inv), -127, 127).astype(np.float64) * (amax / np.float32(127.0)).astype(np.float64)
    W = dense.cpu().numpy().astype(np.float64)
    gmax = np.abs(b).reshape(X.shape[0], -1, 256).max(-1).sum(-1) * 256.0
    return q.reshape(X.shape[0], -1) @ W.T, 2.0 ** -19 * np.outer(gmax, np.abs(W).max(1))


def _gemm(kd, w, X, dtype=torch.float32):
    Y = torch.full((X.shape[0], w.rows), float("nan"), dtype=dtype, device=DEV)
    ws = torch.zeros(kd.quant_gemm_workspace_bytes(*X.shape), dtype=torch.uint8, device=DEV)
    kd.quant_gemm(X.to(DEV), w, Y, ws)
    torch.cuda.synchronize()
    assert kd.device_status() == 0
    return Y


# one row tile per CTA: fewer rows than a tile, one past it, odd row counts; 8-row steps of the activation rows and
# one past each; one super-block and odd numbers of them. Last two: two row tiles and 64-row groups.
@pytest.mark.parametrize("N,K,M", [(1, 256, 4), (33, 256, 8), (97, 512, 9), (128, 768, 17), (129, 1280, 25), (300, 512, 31),
                                   (257, 256, 32), (130, 768, 33), (9600, 256, 200), (19001, 768, 65)])
def test_gemm_edges(kd, N, K, M):
    w = kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(O.Q4_K, N, K, N + M, scale_bits=0x1C00), O.Q4_K, N, K, DEV)
    g = torch.Generator().manual_seed(M)
    X = torch.randn(M, K, generator=g)
    X[:, ::40] *= 30.0                       # blocks of very different scale inside a group
    X[M // 2, :] = 0.0                       # a row without a scale
    X[0, 32:64] = 0.0
    want, bound = _exact(kd, w, X)
    got = _gemm(kd, w, X).cpu().numpy().astype(np.float64)
    assert np.all(np.abs(got - want) <= bound)
    assert torch.equal(_gemm(kd, w, X, torch.bfloat16), _gemm(kd, w, X).to(torch.bfloat16))


def test_a_non_finite_row_stays_alone(kd):
    N, K, M = 200, 512, 12
    w = kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(O.Q4_K, N, K, 3, scale_bits=0x1C00), O.Q4_K, N, K, DEV)
    X = torch.randn(M, K, generator=torch.Generator().manual_seed(1))
    clean = _gemm(kd, w, X)
    X[5, 300] = float("inf")
    got = _gemm(kd, w, X)
    keep = [m for m in range(M) if m != 5]
    assert torch.equal(got[keep], clean[keep]) and bool(torch.isnan(got[5]).all())


@pytest.mark.parametrize("T,E,S", [(100, 4, 2), (7, 5, 1), (65, 1, 1)])   # runs past 32 rows take 64-row groups
@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
def test_moe_groups(kd, port, T, E, S, x_dtype):
    H, F = 512, 768                          # three super-blocks of the down projection
    mk = lambda r, c, s: [kd.ggml_pack.synth_weight(O.Q4_K, r, c, s + e, std=0.05) for e in range(E)]
    gate, up, down = mk(F, H, 1), mk(F, H, 100), mk(H, F, 200)
    tab = lambda lst, r, c: kd.make_quant_weight_table([kd.QuantWeight.from_numpy(a, O.Q4_K, r, c, DEV) for a in lst])
    rng = np.random.default_rng(T)
    X = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).to(x_dtype)
    idx = np.stack([rng.permutation(E)[:S] for _ in range(T)]).astype(np.int32)
    idx[1:T // 2, 0] = 0                     # one expert with a long run (a token may name it twice)
    wts = rng.random((T, S)).astype(np.float32)
    ws = torch.zeros(kd.moe_ffn_workspace_bytes(T, S, H, F, E), dtype=torch.uint8, device=DEV)
    Y = torch.full((T, H), float("nan"), dtype=torch.float32, device=DEV)
    kd.moe_ffn(X.to(DEV), tab(gate, F, H), tab(up, F, H), tab(down, H, F), torch.from_numpy(idx).to(DEV),
               torch.from_numpy(wts).to(DEV), Y, ws)
    torch.cuda.synchronize()
    assert kd.device_status() == 0
    al = lambda lst: [O.aligned_copy(a) for a in lst]
    ref = port.moe_ffn_int8(X.float().numpy(), al(gate), al(up), al(down), idx, wts, F, (O.Q4_K,) * 3,
                            bf16=(x_dtype == torch.bfloat16))
    assert np.abs(Y.cpu().numpy() - ref).max() <= 1e-3 * np.abs(ref).max()
