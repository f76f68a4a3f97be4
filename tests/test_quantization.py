"""Weight-only quantisation: every format round-trips within its expected error, the CUDA dequant / GEMV kernels
agree with the PyTorch reference, and a quantised model still generates the same greedy tokens as its dequantised
twin."""

import pytest
import torch

from easydel_b200.layers.quantization import (FORMATS, EasyDeLQuantizationConfig, EasyQuantizer, QuantizedLinear,
                                              dequantize_reference, quantize, quantized_matmul)

TOL = {"int8": 0.02, "a8bit": 0.02, "a4bit": 0.2, "affine": 0.2, "nf4": 0.2, "mxfp4": 0.3, "nvfp4": 0.25,
       "mxfp8": 0.08, "nvfp8": 0.08}


@pytest.mark.parametrize("fmt", sorted(FORMATS))
def test_roundtrip_error(fmt):
    torch.manual_seed(0)
    w = torch.randn(64, 256) * 0.05
    q = quantize(w, fmt)
    back = dequantize_reference(q)
    rel = (back - w).norm() / w.norm()
    assert rel < TOL[fmt], (fmt, float(rel))
    assert q.nbytes() < w.numel() * 2
    x = torch.randn(3, 256)
    y = quantized_matmul(x, q)
    assert torch.allclose(y, x @ back.t(), atol=1e-4)


def test_quantizer_replaces_linears_and_keeps_outputs_close():
    from easydel_b200.modules.llama import LlamaConfig, LlamaForCausalLM

    cfg = LlamaConfig(vocab_size=128, hidden_size=64, intermediate_size=128, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, max_position_embeddings=64)
    torch.manual_seed(0)
    model = LlamaForCausalLM(cfg, dtype=torch.float32, param_dtype=torch.float32).eval()
    ids = torch.randint(0, 128, (2, 16))
    with torch.no_grad():
        ref = model(input_ids=ids).logits
    model.quantize(EasyDeLQuantizationConfig("int8", block_size=64))
    n = sum(isinstance(m, QuantizedLinear) for m in model.modules())
    assert n == 2 * 4 and not isinstance(model.lm_head, QuantizedLinear)
    with torch.no_grad():
        got = model(input_ids=ids).logits
    assert (got - ref).abs().max() < 0.05 * ref.abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["nf4", "int8"])
@pytest.mark.parametrize("K,M", [(47104, 16), (47232, 16), (94208, 8), (94336, 8), (94336, 1)])
def test_products_at_the_limit_of_shared_memory(fmt, K, M):
    torch.manual_seed(0)
    block = 64 if fmt == "nf4" else 128
    q = quantize(torch.randn(24, K, device="cuda") * 0.05, EasyDeLQuantizationConfig(fmt, block_size=block))
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    ref = x.double() @ dequantize_reference(q).double().t()
    # above the limit weights are rounded to bf16 first: 2^-9 of each product, adding up as a random walk
    assert (quantized_matmul(x, q).double() - ref).abs().max() <= 2.0 ** -7 * ref.abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,block", [("nf4", 64), ("nf4", 128), ("nf4", 96), ("affine", 32), ("a4bit", 64), ("mxfp4", None),
                                       ("int8", 128), ("int8", 48), ("a8bit", 32), ("mxfp8", None), ("nvfp8", None)])
@pytest.mark.parametrize("N,K", [(5, 96), (17, 288), (130, 1152), (1000, 6240)])
@pytest.mark.parametrize("odd", [False, True])
def test_fused_product_at_its_edges(fmt, block, N, K, odd):
    """The fused product of a few rows: ragged weight rows and reductions, groups within, across and beyond a lane's 16 bytes
    of codes, 1 to 16 activation rows, and the expansion behind more; ``odd``: codes that start on 4 bytes only, strided
    activations, a bias."""
    from easydel_b200.layers.quantization import QuantizedTensor

    if block is not None and K % block:
        K = max(1, K // block) * block
    torch.manual_seed(N)
    q = quantize(torch.randn(N, K, device="cuda") * 0.05, EasyDeLQuantizationConfig(fmt, block_size=block))
    if odd:
        raw = torch.empty(q.codes.numel() + 4, dtype=torch.uint8, device="cuda")
        codes = raw[4:].view(q.codes.shape)
        codes.copy_(q.codes)
        q = QuantizedTensor(codes, q.scales, q.zeros, q.lut, q.bits, q.group, q.shape, q.fmt)
    w = dequantize_reference(q).double()
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16) if odd else None
    for M in (1, 3, 8, 9, 16):
        x = torch.randn(M, K + (3 if odd else 0), device="cuda").to(torch.bfloat16)[:, :K]
        y = quantized_matmul(x, q, bias)
        ref = x.double() @ w.t() + (0 if bias is None else bias.double())
        # bf16 rounds the result by 2^-9; values keep 16 bits (2^-17 each), sums are fp32
        tol = 2.0 ** -8 * ref.abs() + 2.0 ** -16 * (x.double().abs() @ w.abs().t())
        assert ((y.double() - ref).abs() <= tol).all(), M
    assert torch.equal(q.dequantize(), dequantize_reference(q).to(torch.bfloat16))
    x = torch.randn(17, K, device="cuda").to(torch.bfloat16)
    ref = x.double() @ w.t() + (0 if bias is None else bias.double())
    # weights are rounded to bf16 as well: 2^-9 of each product
    tol = 2.0 ** -8 * ref.abs() + 2.0 ** -9 * 1.01 * (x.double().abs() @ w.abs().t())
    assert ((quantized_matmul(x, q, bias).double() - ref).abs() <= tol).all()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,block", [("nf4", 64), ("a4bit", 32), ("mxfp4", None), ("int8", 128), ("a8bit", 64)])
@pytest.mark.parametrize("N,K", [(60003, 256), (45000, 1152), (38000, 3584)])
def test_fused_product_of_more_rows_than_a_round(fmt, block, N, K):
    """Weight rows beyond what all SMs take at once: CTAs that go over several row tiles, the last ones past the end."""
    torch.manual_seed(N)
    q = quantize(torch.randn(N, K, device="cuda") * 0.05, EasyDeLQuantizationConfig(fmt, block_size=block))
    w = dequantize_reference(q)
    for M in (1, 5, 8):
        x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
        bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
        ref = x.double() @ w.double().t() + bias.double()
        tol = 2.0 ** -8 * ref.abs() + 2.0 ** -16 * (x.double().abs() @ w.double().abs().t())     # as above
        assert ((quantized_matmul(x, q, bias).double() - ref).abs() <= tol).all(), M


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17])
def test_gradients_pass_through_a_quantised_product_of_any_rows(M):
    torch.manual_seed(M)
    q = quantize(torch.randn(64, 256, device="cuda") * 0.05, "nf4")
    x = torch.randn(M, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    dy = torch.randn(M, 64, device="cuda").to(torch.bfloat16)
    (quantized_matmul(x, q).float() * dy).sum().backward()
    want = dy.double() @ dequantize_reference(q).to(torch.bfloat16).double()
    assert ((x.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()      # one rounding to bf16


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["int8", "a4bit", "nf4", "mxfp4", "nvfp4", "mxfp8", "nvfp8"])
@pytest.mark.parametrize("M", [1, 5, 8, 64])
def test_cuda_kernels_match_reference(fmt, M):
    torch.manual_seed(1)
    N, K = 1000 if fmt != "nvfp8" else 512, 1024
    w = (torch.randn(N, K) * 0.05).cuda()
    q = quantize(w, fmt)
    ref_w = dequantize_reference(q)
    got_w = q.dequantize(torch.bfloat16)
    assert torch.allclose(got_w.float(), ref_w.to(torch.bfloat16).float(), atol=1e-6)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    y = quantized_matmul(x, q, bias)
    ref = x.float() @ ref_w.t() + bias.float()
    assert (y.float() - ref).abs().max() < 2e-2 * ref.abs().max().clamp_min(1.0)


def test_straight_through_and_qat_linear():
    """Fake quantisation for training: forward value = quantise -> dequantise, gradient = identity; a wrapped model
    trains its full-precision weights and converts to quantised linears whose output it already produced."""
    import torch
    from torch import nn

    from easydel_b200.layers import quantization as Q

    torch.manual_seed(0)
    w = torch.randn(8, 256, requires_grad=True)
    wq = Q.straight_through(w, "nf4")
    ref = Q.dequantize_reference(Q.quantize(w.detach(), "nf4"))
    assert torch.allclose(wq, ref) and not torch.equal(wq, w)
    (wq * torch.arange(256.0)).sum().backward()
    assert torch.allclose(w.grad, torch.arange(256.0).expand(8, 256))
    for fn in (Q.straight_through_8bit, Q.straight_through_mxfp4, Q.straight_through_mxfp8, Q.straight_through_nvfp8):
        assert fn(w).shape == w.shape
    b = Q.straight_through_1bit(w)
    assert torch.allclose(b.abs(), w.detach().abs().mean(-1, keepdim=True).expand_as(w))

    model = nn.Sequential(nn.Linear(256, 128), nn.ReLU(), nn.Linear(128, 8))
    quantizer = Q.EasyQuantizer("nf4", pattern=r".*")
    quantizer.apply_qat(model)
    assert model.qat_summary["modules"] == 2 and isinstance(model[0], Q.QATLinear)
    x = torch.randn(16, 256)
    before = model[0].inner.weight.detach().clone()
    opt = torch.optim.SGD(model.parameters(), lr=0.1)
    loss = model(x).pow(2).mean()
    loss.backward()
    opt.step()
    assert not torch.equal(model[0].inner.weight, before)          # the full-precision weight moved
    y_qat = model(x)
    quantizer.finalize_qat(model)
    assert isinstance(model[0], Q.QuantizedLinear)
    assert torch.allclose(model(x), y_qat, atol=1e-4)
