"""Quantised linears: layouts (CPU) and the tcgen05 dequant-GEMM (GPU) against dequantise-then-matmul in fp32."""
import numpy as np
import pytest
import torch

from eredu_b200.lib import _eredu_host as H
from eredu_b200.ops.quant import (QuantLinear, affine_quantize_tensor, codes_to_kernel4, unpack_bitstream)


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_unpack_bitstream_matches_host_codec(bits):
    rng = np.random.default_rng(bits)
    w = (rng.standard_normal((6, 256)) * 0.1).astype(np.float32)
    packed, scales, biases = H.affine_quantize(w, bits, 64 if bits != 6 else 16, "bf16")
    codes = unpack_bitstream(torch.from_numpy(packed.astype(np.int64)).to(torch.int32), bits)
    assert np.array_equal(codes.numpy(), H.unpack_codes(packed, bits))


def test_kernel_layout_round_trip_and_device_quantizer_matches_host():
    torch.manual_seed(0)
    w = torch.randn(16, 512) * 0.05
    codes, s, b = affine_quantize_tensor(w, 4, 64)
    ql = QuantLinear(codes, s, b, 4, 64, "cpu")
    assert torch.equal(ql.codes(), codes)
    assert ql.wq.shape == (1, 8, 512)          # one 16-row tile, eight 64-column blocks of 512 bytes
    # tile (0, kb) holds rows 0..15 x columns 64 kb .. 64 kb + 63: row r of the tile is 32 bytes at offset 32 r
    from eredu_b200.ops.quant import untile_kernel4

    rows = untile_kernel4(ql.wq, 16)
    assert torch.equal(ql.wq[0, 3].view(16, 32), rows[:, 96:128])
    hp, hs, hb = H.affine_quantize(w.numpy(), 4, 64, "bf16")
    assert np.array_equal(H.unpack_codes(hp, 4), codes.numpy())
    assert np.allclose(hs, s.float().numpy()) and np.allclose(hb, b.float().numpy())
    deq = ql.dequantize()
    assert float((deq - w).abs().max()) < 0.02
    x = torch.randn(3, 512)
    assert torch.allclose(ql(x), x @ deq.t(), atol=1e-4)
    # row / column slices and mixed-width fusion keep every value
    a = ql.slice_rows(4, 12).slice_cols(128, 384)
    assert torch.equal(a.dequantize(), deq[4:12, 128:384])
    w2 = torch.randn(40, 512) * 0.05
    big = QuantLinear(*affine_quantize_tensor(w2, 4, 64), 4, 64, "cpu")
    d2 = big.dequantize()
    assert big.wq.shape == (3, 8, 512)
    assert torch.equal(big.slice_rows(16, 40).dequantize(), d2[16:]) and torch.equal(big.slice_rows(16, 32).dequantize(), d2[16:32])
    assert torch.equal(big.slice_rows(5, 37).dequantize(), d2[5:37])
    both = QuantLinear.concat_rows([big, ql])                  # 40 rows are no whole number of tiles: repacked
    assert both.out_features == 56 and torch.equal(both.dequantize(), torch.cat((d2, deq)))
    even = QuantLinear.concat_rows([ql, big])
    assert torch.equal(even.dequantize(), torch.cat((deq, d2))) and even.wq.shape == (4, 8, 512)
    assert big.decode_table().shape == (3, 8, 16) and big.slice_cols(64, 192).decode_table().shape == (3, 2, 16)
    c8, s8, b8 = affine_quantize_tensor(w[:8], 6, 16)
    fused = QuantLinear.concat_rows([ql, QuantLinear(c8, s8, b8, 6, 16, "cpu")])
    assert fused.kbits == 8 and fused.group == 16
    assert torch.equal(fused.dequantize()[:16], deq)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,group", [(4, 64), (4, 32), (4, 128), (8, 32), (6, 16), (4, 16)])
@pytest.mark.parametrize("M", [1, 7, 32, 50, 128, 300])
def test_qgemm_matches_dequantized_matmul(bits, group, M):
    torch.manual_seed(bits * 1000 + group + M)
    N, K = 640, 1024
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    ql = QuantLinear.from_dense(w, bits, group)
    x = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    res = torch.randn(M, N, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    y = ql(x, bias=bias, residual=res)
    deq = ql.dequantize(torch.float32)
    ref = x.float() @ deq.t() + bias.float() + res.float()
    rel = float((y.float() - ref).norm() / ref.norm())
    assert rel < 1e-2, rel
    from eredu_b200.ops import native
    native.check_status(torch.device("cuda", torch.cuda.current_device()))


@pytest.mark.gpu
@pytest.mark.parametrize("wk,ns", [(1, 1), (2, 1), (8, 1), (1, 2), (4, 4), (8, 8), (0, 0)])
@pytest.mark.parametrize("M,group,gated,exact", [(1, 64, False, 0), (8, 64, True, 0), (5, 32, False, 0), (7, 128, True, 0),
                                                 (8, 16, False, 0), (3, 64, True, 1), (6, 128, False, 1)])
def test_decode_kernel_every_k_split_against_fp32(wk, ns, M, group, gated, exact):
    """The register-resident decode kernel (mma.sync over codes dequantised in registers) with K split over the warps
    of a CTA, over a cluster, both, or as the host picks it (0, 0); plain and SwiGLU epilogues; ragged row count; the
    accumulator-side affine map (groups of 64 / 128) and the in-register bf16 dequantisation (small groups, or forced)."""
    from eredu_b200.ops.native import check_status, lib, ptr, status_word, stream_ptr

    torch.manual_seed(wk * 100 + ns * 10 + M)
    N, K = (2 * 336 if gated else 650), 1536 + 128
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    ql = QuantLinear.from_dense(w, 4, group)
    x = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    res = None if gated else torch.randn(M, N, device="cuda").bfloat16()
    n_out = N // 2 if gated else N
    y = torch.full((M, n_out), float("nan"), dtype=torch.bfloat16, device="cuda")
    code = lib().eredu_qgemv4(ptr(x), ptr(ql.wq), ptr(ql.decode_table()), ptr(y), ptr(res), ptr(bias), M, N, K, x.stride(0),
                              y.stride(0), 0 if res is None else res.stride(0), group, 0, int(gated), 0.0, wk, ns, exact, 148,
                              None, ptr(status_word(x.device)), stream_ptr(x.device))
    assert code == 0
    check_status(x.device)
    lin = x.float() @ ql.dequantize(torch.float32).t() + bias.float()
    ref = torch.nn.functional.silu(lin[:, :n_out]) * lin[:, n_out:] if gated else lin + res.float()
    rel = float((y.float() - ref).norm() / ref.norm())
    assert rel < 1e-2, rel
    # the public call takes the same kernel for these sizes and agrees with the explicit launch
    pub = ql.gated(x, bias=bias) if gated else ql(x, bias=bias, residual=res)
    assert float((pub.float() - y.float()).abs().max()) <= 0.05 * float(ref.abs().max())


@pytest.mark.gpu
def test_qgemm_shapes_of_the_70b_shard_and_fp32_out():
    torch.manual_seed(0)
    for N, K in ((1280, 8192), (8192, 1024), (7168, 8192), (8192, 3584)):
        w = (torch.randn(N, K, device="cuda") * 0.02).bfloat16()
        ql = QuantLinear.from_dense(w, 4, 64)
        for M in (1, 8):
            x = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
            y = ql(x, out_dtype=torch.float32)
            ref = x.float() @ ql.dequantize().t()
            assert float((y - ref).norm() / ref.norm()) < 1e-2
        assert abs(ql.nbytes() / (N * K) - (0.5 + 4 / 64)) < 1e-6


@pytest.mark.gpu
def test_gguf_q4k_q6k_model_runs_on_native_codes(tmp_path):
    import dataclasses

    from eredu_b200.api import LoadedModel, ModelLoadOptions
    from eredu_b200.formats import checkpoint as ck
    from eredu_b200.models import config as C
    from eredu_b200.models.llama import random_state

    cfg = dataclasses.replace(C.tiny_llama(), hidden_size=512, num_attention_heads=8, num_key_value_heads=2, head_dim=64,
                              intermediate_size=1024, vocab_size=1024, num_hidden_layers=2, tie_word_embeddings=False)
    sd = random_state(cfg, seed=0, std=0.05)
    path = tmp_path / "m.gguf"
    ck.save_gguf_checkpoint(path, cfg, sd, type_for=lambda n: "Q6_K" if ("attn_v" in n or "ffn_down" in n) else
                            ("F32" if ("token_embd" in n or n.startswith("output")) else "Q4_K"))
    native = LoadedModel.load(path, ModelLoadOptions(device="cuda", max_batch=1, max_seq_len=128, native_gguf=True))
    dense = LoadedModel.load(path, ModelLoadOptions(device="cuda", max_batch=1, max_seq_len=128, native_gguf=False))
    assert "qkv" in native.model.layers[0].qlin and native.model.layers[0].qlin["qkv"].kbits == 8
    assert native.model.layers[0].qlin["o"].kbits == 4 and not dense.model.layers[0].qlin
    prompt = list(range(3, 40))
    a, b = native.prefill_logits(prompt), dense.prefill_logits(prompt)
    rel = float((a - b).norm() / b.norm())
    assert rel < 0.05 and torch.nn.functional.cosine_similarity(a, b, dim=0) > 0.995


@pytest.mark.parametrize("shape, dtype", [((300, 192), torch.bfloat16), ((300, 320), torch.bfloat16), ((4, 192), torch.bfloat16), ((300, 256), torch.float32)])
def test_gated_projection_refuses_rows_of_another_width_or_type(shape, dtype):
    """Before anything is launched: the kernels take the width from the rows."""
    class Rows:
        is_cuda = True

        def stride(self, dim):
            return (self.shape[1], 1)[dim]

    x = Rows()
    x.shape, x.dtype = shape, dtype
    ql = QuantLinear.from_dense(torch.randn(128, 256), 4, 64)
    with pytest.raises(AssertionError):
        ql.gated(x)
