"""The split-fp16 tensor-core kernel (csrc/kdnn_split.cuh) at the edges of its tiles, against float64.

Bound of the edge cases (indexing, masks, remainders; far wider than the arithmetic needs): |error| <= 2^-19 *
max|W row| * sum_k (group maximum of |x|). How exact the sums are is held by test_error_by_distribution and
test_down_product_of_known_activations, to relative 2-norms that a lost fp16 part misses by a factor of a hundred
(test_bounds_notice_a_lost_part shows it on the CPU)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

gpu = pytest.mark.gpu
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


@pytest.fixture
def split_kernel(kd):
    """The kernel under test whatever the size rules of the default kind prefer."""
    prev = kd.tile_kind(kd.TILE_SPLIT)
    yield
    kd.tile_kind(prev)


# one row tile per CTA: fewer rows than a tile, one past it, odd row counts; 8-row steps of the activation rows and
# one past each; one super-block and odd numbers of them. Last two: two row tiles and 64-row groups.
@gpu
@pytest.mark.parametrize("N,K,M", [(1, 256, 4), (33, 256, 8), (97, 512, 9), (128, 768, 17), (129, 1280, 25), (300, 512, 31),
                                   (257, 256, 32), (130, 768, 33), (9600, 256, 200), (19001, 768, 65)])
def test_gemm_edges(kd, split_kernel, N, K, M):
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


@gpu
def test_a_non_finite_row_stays_alone(kd, split_kernel):
    N, K, M = 200, 512, 12
    w = kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(O.Q4_K, N, K, 3, scale_bits=0x1C00), O.Q4_K, N, K, DEV)
    X = torch.randn(M, K, generator=torch.Generator().manual_seed(1))
    clean = _gemm(kd, w, X)
    X[5, 300] = float("inf")
    got = _gemm(kd, w, X)
    keep = [m for m in range(M) if m != 5]
    assert torch.equal(got[keep], clean[keep]) and bool(torch.isnan(got[5]).all())


@gpu
@pytest.mark.parametrize("T,E,S", [(100, 4, 2), (7, 5, 1), (65, 1, 1)])   # runs past 32 rows take 64-row groups
@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
def test_moe_groups(kd, port, split_kernel, T, E, S, x_dtype):
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


def _least_workspace(M, K):
    up = lambda v: (v + 255) // 256 * 256
    row = up(K + 24 * (K // 32) + 48 * ((K // 32 + 7) // 8))
    return 512 + up(M * 4) + up((M + 31) // 32 * 16) + M * max(K // 64 * 96, row)


@gpu
@pytest.mark.parametrize("fmt,M,kind", [(O.Q4_K, 5, 2), (O.Q4_K, 8, 2), (O.Q4_K, 9, 1), (O.Q4_K, 70, 1), (O.Q6_K, 4, 0), (O.Q6_K, 9, 0)])
def test_a_workspace_of_the_integer_kernels_size_is_served_by_them(kd, fmt, M, kind):
    N, K = 130, 768
    w = kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(fmt, N, K, M, scale_bits=0x1C00), fmt, N, K, DEV)
    X = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(DEV)
    out = []
    for tile, nbytes in ((kd.TILE_AUTO, _least_workspace(M, K)), (kind, kd.quant_gemm_workspace_bytes(M, K))):
        prev = kd.tile_kind(tile)
        try:
            Y = torch.full((M, N), float("nan"), device=DEV)
            big = torch.full((nbytes + 256,), 7, dtype=torch.uint8, device=DEV)
            kd.quant_gemm(X, w, Y, big[:nbytes])
            torch.cuda.synchronize()
            assert bool((big[nbytes:] == 7).all())
        finally:
            kd.tile_kind(prev)
        out.append(Y)
    assert torch.equal(out[0], out[1])


# ---- how exact the sums are --------------------------------------------------------------------------
def _rows(kind, M, K, g):
    """Activation rows, and the columns whose weights are zero."""
    x, zero = torch.randn(M, K, generator=g), torch.zeros(K, dtype=torch.bool)
    if kind == "outliers":
        x[:, ::64] *= 8.0
    elif kind == "one sign":
        x = x.abs()
    elif kind == "squared relu":
        x = x.clamp(min=0.0) ** 2
    elif kind == "constant":
        x = torch.ones_like(x)
    elif kind == "far from zero":
        x = 3.0 + x
    elif kind == "wide":
        x = torch.exp(2.0 * x)
    elif kind.startswith("spike"):      # a block far above its group whose own weights are zero
        zero.view(-1, 256)[:, 96:128] = True
        x[:, zero] *= float(kind.split()[1])
    return x, zero


ROWS = ["normal", "outliers", "one sign", "squared relu", "constant", "far from zero", "wide", "spike 30", "spike 1000",
        "spike 10000"]


def _rel(got, want):
    return float(np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want))


@gpu
@pytest.mark.parametrize("one_sign_weights", [False, True])
@pytest.mark.parametrize("kind", ROWS)
def test_error_by_distribution(kd, kind, one_sign_weights):
    """fp32 outputs against float64: at most 1e-6, and at most 1.25 times what the mma.sync kernel shows on the same
    rows, whose per-32 dots are exact integers (measured 0.1 to 0.7e-6 against 0.1 to 6e-6), but not below 2e-7: per group
    three sums are cut to 24 bits (up to 2^-23, 0.58 of that root mean square) and four fp32 roundings follow, 1.4e-7 of
    the group. 24 rows take the kernel of one row tile, 650 rows that of two and 64-row groups."""
    for N, K, M in ((256, 2048, 24), (4096, 1024, 650)):
        g = torch.Generator().manual_seed(7)
        x, zero = _rows(kind, M, K, g)
        W = torch.randn(N, K, generator=g).numpy() * 0.02
        W = np.abs(W) if one_sign_weights else W
        W[:, zero.numpy()] = 0.0
        w = kd.QuantWeight.from_numpy(kd.ggml_pack.quantize(O.Q4_K, W.astype(np.float32)), O.Q4_K, N, K, DEV)
        want, _ = _exact(kd, w, x)
        err = {}
        for tile in (kd.TILE_SPLIT, kd.TILE_MMA_SYNC):
            prev = kd.tile_kind(tile)
            try:
                err[tile] = _rel(_gemm(kd, w, x).cpu().numpy(), want)
            finally:
                kd.tile_kind(prev)
        assert err[kd.TILE_SPLIT] <= min(1e-6, max(2e-7, 1.25 * err[kd.TILE_MMA_SYNC])), (N, K, M, err)


@gpu
@pytest.mark.parametrize("T", [20, 40])
def test_down_product_of_known_activations(kd, split_kernel, T):
    """One expert with weight 1: the down product (128-element groups) against float64 of the activations as
    quantized. A gate or up product that rounds the other way turns an activation by one int8 step in a few rows, so the
    bound is on three rows of four: 1e-6."""
    H, F = 512, 1024
    mk = lambda r, c, s: kd.QuantWeight.from_numpy(kd.ggml_pack.synth_weight(O.Q4_K, r, c, s, std=0.05), O.Q4_K, r, c, DEV)
    gate, up, down = mk(F, H, 1), mk(F, H, 2), mk(H, F, 3)
    x = torch.randn(T, H, generator=torch.Generator().manual_seed(T))
    a, b = _exact(kd, gate, x)[0], _exact(kd, up, x)[0]
    act = (a / (1.0 + np.exp(-a)) * b).astype(np.float32)
    want, _ = _exact(kd, down, torch.from_numpy(act))
    Y = torch.full((T, H), float("nan"), dtype=torch.float32, device=DEV)
    ws = torch.zeros(kd.moe_ffn_workspace_bytes(T, 1, H, F, 1), dtype=torch.uint8, device=DEV)
    tab = lambda q: kd.make_quant_weight_table([q])
    kd.moe_ffn(x.to(DEV), tab(gate), tab(up), tab(down), torch.zeros(T, 1, dtype=torch.int32, device=DEV),
               torch.ones(T, 1, device=DEV), Y, ws)
    torch.cuda.synchronize()
    got = Y.cpu().numpy().astype(np.float64)
    rows = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert np.quantile(rows, 0.75) <= 1e-6, np.sort(rows)


def _split(x, parts):
    """The split form of fp32 rows as float64, with both fp16 parts or the first alone (split_store_lane8, K = 256 groups)."""
    b = x.reshape(x.shape[0], -1, 8, 32)
    amax = np.abs(b).max(-1, keepdims=True)
    inv = np.divide(np.float32(127.0), amax, out=np.zeros_like(amax), where=amax > 0)
    q, d = np.clip(np.rint(b * inv), -127, 127), amax / np.float32(127.0)
    D = d.max(2, keepdims=True)
    r = np.float32(256.0) * (d / D)
    v = (q * r).astype(np.float32)
    need = np.maximum(600.0 * np.sqrt((v.astype(np.float64) ** 2).sum((2, 3), keepdims=True)),
                      768.0 * np.abs(q.sum(-1, keepdims=True) * r / 16.0).sum(2, keepdims=True)) / 2.0 ** 24
    u = 2.0 ** np.ceil(np.log2(np.clip(need, 2.0, 32.0)))
    step = np.minimum(u, np.maximum(2.0 ** np.floor(np.log2(np.maximum(r, 1e-30))) / 8.0, 2.0 ** -24))
    hi = (np.rint(v / step) * step).astype(np.float16)
    mid = (v - hi.astype(np.float32)).astype(np.float16)
    out = hi.astype(np.float64) + (mid.astype(np.float64) if parts == 2 else 0.0)
    return (out * D.astype(np.float64) / 256.0).reshape(x.shape), (q.astype(np.float64) * d.astype(np.float64)).reshape(x.shape)


@pytest.mark.parametrize("kind", ROWS)
def test_bounds_notice_a_lost_part(kind):
    """The arithmetic of the bounds above: both parts stay a factor of five below 1e-6, one part alone misses it (a
    constant row is a multiple of every step, there one part is exact)."""
    g = torch.Generator().manual_seed(11)
    x, zero = _rows(kind, 8, 1024, g)
    W = np.random.default_rng(1).standard_normal((64, 1024)) * 0.02
    W[:, zero.numpy()] = 0.0
    both, exact = _split(x.numpy(), 2)
    one, _ = _split(x.numpy(), 1)
    want = exact @ W.T
    assert _rel(both @ W.T, want) <= 2e-7
    assert kind == "constant" or _rel(one @ W.T, want) >= 2e-5
