"""One token through the expert feed-forward (the two token kernels of csrc/kdnn_moe.cu) against the general path
(tile kind 0: slot sort, quantizer launches, dp4a kernels, combine), which does the same arithmetic in another order.

Bound: the gate and up sums differ by fp32 rounding, which turns an activation by one int8 step (1/127 of its block's
largest) in places, and outputs are at least as large as one such term: 1/127 of the largest output."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# fewer items than lanes, as many, one more; a row count that leaves the last CTA short (256 = 16 x 16, 768 = 96 x 8);
# the largest quantized slots that fit 48 KB of shared memory (4 x 8192) and the first that do not (4 x 8448); eight
# slots of that size, which go through the tiles
@pytest.mark.parametrize("H,F,S", [(256, 256, 1), (2048, 768, 8), (2304, 512, 3), (512, 8192, 4), (512, 8448, 4), (512, 4096, 8),
                                   (512, 4352, 8)])
@pytest.mark.parametrize("fmts", [(O.Q4_K, O.Q4_K), (O.Q4_K, O.Q6_K), (O.Q5_K, O.Q8_0), (O.Q6_K, O.Q5_K)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_token_equals_general_path(kd, fmts, H, F, S, dtype):
    E = 9

    def table(fmt, rows, cols, seed):
        return kd.make_quant_weight_table(
            [kd.QuantWeight.from_numpy(kd.ggml_pack.random_payload(fmt, rows, cols, seed + e, scale_bits=0x1400), fmt, rows, cols, DEV)
             for e in range(E)], "w")

    gate, up, down = table(fmts[0], F, H, 1), table(fmts[0], F, H, 100), table(fmts[1], H, F, 200)
    g = torch.Generator().manual_seed(H + F + S)
    X = torch.randn(1, H, generator=g).to(dtype).to(DEV)
    idx = torch.randperm(E, generator=g)[:S].to(torch.int32)
    wts = torch.rand(1, S, generator=g)
    if S > 2:
        idx[1] = idx[0]          # one expert twice
        wts[0, 2] = 0.0          # a slot without weight
    if S > 4:
        idx[3], idx[4] = -1, E   # slots outside the table
    idx, wts = idx.reshape(1, S).to(DEV), wts.to(DEV)
    out = []
    for kind in (3, 0):
        prev = kd.tile_kind(kind)
        try:
            Y = torch.full((1, H), float("nan"), dtype=torch.float32, device=DEV)
            ws = torch.zeros(kd.moe_ffn_workspace_bytes(1, S, H, F, E), dtype=torch.uint8, device=DEV)
            kd.moe_ffn(X, gate, up, down, idx, wts, Y, ws)
            torch.cuda.synchronize()
        finally:
            kd.tile_kind(prev)
        out.append(Y.cpu().numpy().astype(np.float64))
    assert np.isfinite(out[1]).all() and np.abs(out[1]).max() > 0
    assert np.abs(out[0] - out[1]).max() <= np.abs(out[1]).max() / 127


def _product(kd, w, x):
    """float64 W . q(x) with the int8-quantized row; weights from the bit-exact dequantizer."""
    dense = torch.empty((w.rows, w.cols), dtype=torch.float32, device=DEV)
    kd.dequant_to_dense(w, dense)
    b = x.reshape(-1, 32).astype(np.float32)
    amax = np.abs(b).max(-1, keepdims=True)
    inv = np.divide(np.float32(127.0), amax, out=np.zeros_like(amax), where=amax > 0)
    q = np.clip(np.rint(b * inv), -127, 127).astype(np.float64) * (amax / np.float32(127.0)).astype(np.float64)
    return dense.cpu().numpy().astype(np.float64) @ q.reshape(-1)


@pytest.mark.parametrize("fmts", [(O.Q4_K, O.Q4_K), (O.Q4_K, O.Q6_K), (O.Q8_0, O.Q4_K)])
def test_token_against_float64(kd, fmts):
    """fp32 outputs of eight tokens, one expert: relative 2-norm at most 1e-6 for the median token (fp32 sums of at most 768 and
    512 terms; a product that rounds the other way turns an activation by one int8 step in a token here and there). The bf16
    output is the fp32 output rounded once."""
    H, F = 768, 512
    mk = lambda fmt, r, c, s: kd.QuantWeight.from_numpy(kd.ggml_pack.synth_weight(fmt, r, c, s, std=0.05), fmt, r, c, DEV)
    gate, up, down = mk(fmts[0], F, H, 1), mk(fmts[0], F, H, 2), mk(fmts[1], H, F, 3)
    tabs = [kd.make_quant_weight_table([w]) for w in (gate, up, down)]
    idx, wts = torch.zeros(1, 1, dtype=torch.int32, device=DEV), torch.ones(1, 1, device=DEV)
    err = []
    for seed in range(8):
        x = torch.randn(1, H, generator=torch.Generator().manual_seed(seed))
        out = {}
        for dtype in (torch.float32, torch.bfloat16):
            Y = torch.full((1, H), float("nan"), dtype=dtype, device=DEV)
            ws = torch.zeros(kd.moe_ffn_workspace_bytes(1, 1, H, F, 1), dtype=torch.uint8, device=DEV)
            kd.moe_ffn(x.to(DEV), *tabs, idx, wts, Y, ws)
            torch.cuda.synchronize()
            out[dtype] = Y
        assert torch.equal(out[torch.bfloat16], out[torch.float32].to(torch.bfloat16))
        a, b = _product(kd, gate, x.numpy()), _product(kd, up, x.numpy())
        want = _product(kd, down, (a / (1.0 + np.exp(-a)) * b).astype(np.float32))
        err.append(np.linalg.norm(out[torch.float32].cpu().numpy()[0] - want) / np.linalg.norm(want))
    assert np.median(err) <= 1e-6, err
