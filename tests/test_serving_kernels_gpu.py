"""Kernels of the serving path at the edges of their tiles and at the borders between their variants, against fp32 references."""
import pytest
import torch

from eredu_b200 import ops
from eredu_b200.ops import moe as moe_ops
from eredu_b200.ops.native import check_status
from eredu_b200.ops.quant import QuantLinear

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = 2.0 ** -8        # what rounding to bf16 changes at the most, relative to the number


def rel_l2(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


@pytest.fixture(autouse=True)
def _status():
    torch.manual_seed(0)
    yield
    check_status(torch.device("cuda", torch.cuda.current_device()))


@pytest.mark.parametrize("M,n_q,n_kv", [(1, 8, 2), (3, 5, 1), (300, 32, 8), (17, 64, 8)])
@pytest.mark.parametrize("D,rot,interleaved", [(128, 128, False), (64, 64, True), (128, 32, False), (64, 16, True), (64, 24, False), (128, 40, True)])
def test_rotation_and_append_rows(M, n_q, n_kv, D, rot, interleaved):
    """Token counts and head counts around what a CTA takes in one pass; rotated parts that are whole pairs of 16-byte pieces and such that
    are not; rows that are part of wider ones, norms on queries only."""
    wide = torch.randn(M, (n_q + 2 * n_kv) * D + 16, device=DEV).bfloat16()
    qkv = wide[:, :(n_q + 2 * n_kv) * D]
    pos = torch.randint(0, 9000, (M,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(40 * 16, device=DEV)[:M].long()
    slots[M // 2] = -1 if M > 1 else 5
    inv = 1.0 / (10000.0 ** (torch.arange(0, rot, 2, device=DEV).float() / rot))
    qn = torch.rand(D, device=DEV) + 0.5 if M != 3 else None
    kc, vc = (torch.zeros(40, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
    kr, vr = kc.clone(), vc.clone()
    args = dict(rot=rot, interleaved=interleaved, q_norm_w=qn, attn_factor=1.25)
    q = ops.rope_kv(qkv, pos, slots, inv, kc, vc, n_q, n_kv, D, **args)
    ref = ops.rope_kv_ref(qkv.contiguous(), pos, slots, inv, kr, vr, n_q, n_kv, D, **args)
    # sums in another order move a number by one place at the most, and few of them
    assert rel_l2(q, ref) < BF16 and rel_l2(kc, kr) < BF16
    assert torch.equal(vc, vr)


@pytest.mark.parametrize("M", [125, 126, 133, 134])
def test_rotation_of_few_tokens(M):
    """On either side of where a token has a CTA of its own (20 heads of 128 with norms: from 134 tokens on)."""
    test_rotation_and_append_rows(M, 16, 2, 128, 128, False)


@pytest.mark.parametrize("norms", ["none", "queries", "both"])
@pytest.mark.parametrize("D,rot,interleaved", [(128, 128, False), (128, 128, True), (64, 64, False), (64, 48, True), (128, 16, False)])
def test_rotation_gives_the_same_bits_on_either_kernel(D, rot, interleaved, norms):
    """Whole 16-byte pieces, and the same numbers one element further on in rows of odd pitch, which the kernel of single elements takes."""
    M, n_q, n_kv = 700, 12, 2
    width = (n_q + 2 * n_kv) * D
    odd = torch.randn(M, width + 1, device=DEV).bfloat16()
    pos = torch.randint(0, 9000, (M,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(48 * 16, device=DEV)[:M].long()
    inv = 1.0 / (10000.0 ** (torch.arange(0, rot, 2, device=DEV).float() / rot))
    qn = torch.rand(D, device=DEV) + 0.5 if norms != "none" else None
    kn = torch.rand(D, device=DEV) + 0.5 if norms == "both" else None
    outs = []
    for qkv in (odd[:, 1:].contiguous(), odd[:, 1:]):
        kc, vc = (torch.zeros(48, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
        outs.append((ops.rope_kv(qkv, pos, slots, inv, kc, vc, n_q, n_kv, D, rot=rot, interleaved=interleaved, q_norm_w=qn, k_norm_w=kn,
                                 attn_factor=1.25), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("N,K,group", [(16, 64, 64), (650, 320, 32), (8, 1024, 128), (130, 192, 96), (256, 448, 16)])
def test_decoded_weights(N, K, group):
    """K blocks that are no multiple of a warp's four, rows that are no whole tiles, group sizes below, at and above a block."""
    ql = QuantLinear.from_dense((torch.randn(N, K, device=DEV) * 0.05).bfloat16(), 4, group)
    got, want = ql._dense().float(), ql.dequantize(torch.float32)
    assert bool(((got - want).abs() <= 1.001 * BF16 * want.abs()).all())


@pytest.mark.parametrize("M,inter,K,bits", [(257, 320, 512, 4), (300, 72, 192, 4), (513, 128, 256, 8)])
def test_gated_projection_of_prompts(M, inter, K, bits):
    ql = QuantLinear.from_dense((torch.randn(2 * inter, K, device=DEV) * 0.05).bfloat16(), bits, 64)
    x = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    bias = torch.randn(2 * inter, device=DEV).bfloat16()
    w = ql._dense().float()
    y = x.float() @ w.t() + bias.float()
    for limit in (0.0, 1.5):
        ref = moe_ops.gated_act_ref(y[:, :inter], y[:, inter:], limit=limit)
        # without a limit only the result is rounded; with one, gate and up are rounded in between as well
        assert rel_l2(ql.gated(x, bias=bias, limit=limit), ref) < (BF16 if not limit else 3 * BF16)


@pytest.mark.parametrize("M,inter,K", [(512, 2056, 1088), (513, 2048, 2048), (513, 136, 2112), (513, 2056, 1088)])
def test_gated_projection_on_either_side_of_short_sums(M, inter, K):
    test_gated_projection_of_prompts(M, inter, K, 4)


@pytest.mark.parametrize("M", [1, 2, 7, 8])
@pytest.mark.parametrize("N,K,group,gated", [(48, 64, 64, False), (208, 192, 64, False), (2 * 48, 8192, 64, True), (1040, 4096, 128, False),
                                             (2 * 4112, 2048, 32, True), (16, 320, 16, False)])
def test_four_bit_rows_of_few_tokens(M, N, K, group, gated):
    """Row tiles that do not fill a warp's four, K blocks that do not fill a slot of its ring or leave splits without any."""
    ql = QuantLinear.from_dense((torch.randn(N, K, device=DEV) * 0.05).bfloat16(), 4, group)
    x = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    y = x.float() @ ql.dequantize(torch.float32).t()
    ref = moe_ops.gated_act_ref(y[:, :N // 2], y[:, N // 2:]) if gated else y
    got = ql.gated(x) if gated else ql(x)
    # the result is rounded; groups below 64 round the decoded weights too
    assert rel_l2(got, ref) < (BF16 if group >= 64 else 2 * BF16)


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K,group,gated", [(148 * 16, 320, 64, False), (148 * 16 + 16, 320, 64, False), (296 * 32, 128, 32, False),
                                             (296 * 32 + 16, 192, 64, False), (80, 64 * 257, 64, False), (2 * 48, 64 * 258, 32, True),
                                             (2 * 296 * 16, 192, 64, True), (2 * (296 * 16 + 16), 192, 64, True), (296 * 64 + 16, 512, 128, False),
                                             (128, 8192, 64, False)])
def test_four_bit_rows_at_the_borders_of_the_plan(M, N, K, group, gated):
    """Matrices on either side of where a warp takes one, two and four row tiles and where fewer warps, or a cluster, split K."""
    test_four_bit_rows_of_few_tokens(M, N, K, group, gated)


@pytest.mark.parametrize("B,n_q,n_kv,D,splits", [(1, 32, 8, 128, 8), (1, 4, 4, 64, 5), (2, 32, 8, 128, 6), (2, 32, 8, 128, 8), (32, 32, 4, 128, 1),
                                                 (37, 64, 4, 128, 1), (38, 64, 4, 128, 1), (3, 16, 1, 64, 3), (1, 8, 1, 128, 32), (1, 32, 8, 64, 18), (3, 8, 1, 64, 49)])
@pytest.mark.parametrize("length", [1, 16, 17, 128, 129, 1025])
def test_decode_attention_of_one_new_token(B, n_q, n_kv, D, splits, length):
    """Grids on either side of where CTAs have eight warps; contexts that leave splits or warps without a page, new tokens that open a page; one
    sequence whose token is not kept; pages, tables and lengths read ahead of the projection."""
    n_pages = length // 16 + 1
    qkv = torch.randn(B, (n_q + 2 * n_kv) * D, device=DEV).bfloat16()
    kc, vc = (torch.randn(B * n_pages + 1, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
    table = (torch.randperm(B * n_pages, device=DEV) + 1).int().view(B, n_pages)
    lens = torch.full((B,), length, device=DEV, dtype=torch.int32)
    lens[B // 2:] = max(1, length - 5)
    slots = table.gather(1, ((lens - 1) // 16).long()[:, None])[:, 0].long() * 16 + (lens - 1) % 16
    if B > 1:
        slots[1] = -1
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device=DEV).float() / D))
    norm = torch.rand(D, device=DEV) + 0.5
    kr, vr = kc.clone(), vc.clone()
    got = ops.attention_decode_rope(qkv, kc, vc, table, lens, 1, D ** -0.5, lens - 1, slots, inv, n_q, n_kv, D, attn_factor=1.25, q_norm_w=norm,
                                    splits=splits, settled=True)
    q = ops.rope_kv_ref(qkv, lens - 1, slots, inv, kr, vr, n_q, n_kv, D, attn_factor=1.25, q_norm_w=norm)
    ref = ops.attention_ref(q, kr, vr, table, lens, [1] * B, D ** -0.5)
    assert torch.equal(vc, vr) and rel_l2(kc, kr) < BF16
    # queries, probabilities and the result are rounded
    assert rel_l2(got.view(B, -1), ref.view(B, -1)) < 3 * BF16


@pytest.mark.parametrize("M", [5, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("N,K", [(130, 1024), (131, 2048), (512, 1088), (2176, 1024), (4128, 1024), (4736, 1024)])
@pytest.mark.parametrize("odd", [False, True])
def test_split_sums_of_several_tokens(M, N, K, odd):
    """Rows that are no whole quads of columns, residuals whose rows start anywhere, columns beyond the tokens, one CTA and clusters of two, four and
    eight, and the kernel that takes over where K is not split."""
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(2 * N, K, device=DEV) * K ** -0.5).bfloat16()
    bias = torch.randn(N, device=DEV).bfloat16()
    res = torch.randn(M, N + 8, device=DEV).bfloat16()[:, 1:N + 1] if odd else torch.randn(M, N, device=DEV).bfloat16()
    y = x.double() @ w.double().t()
    got, ssq = ops.linear(x, w[:N], bias=bias, residual=res, want_ssq=True)
    assert rel_l2(got, y[:, :N] + bias.double() + res.double()) < BF16
    assert rel_l2(ssq.sum(-1), got.double().square().sum(-1)) < 1e-5
    assert rel_l2(ops.linear(x, w[:N], out_dtype=torch.float32), y[:, :N]) < BF16 / 256
    scale = (got.double().square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    if N % 8 == 0:
        w2 = (torch.randn(2 * 264, N, device=DEV) * N ** -0.5).bfloat16()
        z = (got.double() * scale) @ w2.double().t()
        assert rel_l2(ops.gated_linear(got, w2, 264, row_ssq=ssq, norm_eps=1e-6), moe_ops.gated_act_ref(z[:, :264].float(), z[:, 264:].float())) < BF16


@pytest.mark.parametrize("M", [1, 5, 33, 100])
@pytest.mark.parametrize("parts", [4, 7, 8])
def test_sums_of_squares_that_start_anywhere(M, parts):
    """Partial sums that are part of a larger buffer start on any float."""
    N, K = 264, 1024
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(2 * N, K, device=DEV) * K ** -0.5).bfloat16()
    ssq = torch.rand(M, parts, device=DEV) * 2 * K / parts
    y = x.double() @ w.double().t() * (ssq.double().sum(-1, keepdim=True) / K + 1e-6).rsqrt()
    for at in range(4):
        part = torch.empty(M * parts + 4, device=DEV)[at:at + M * parts].view(M, parts).copy_(ssq)
        assert rel_l2(ops.linear(x, w[:N], row_ssq=part, norm_eps=1e-6), y[:, :N]) < BF16
        assert rel_l2(ops.gated_linear(x, w, N, row_ssq=part, norm_eps=1e-6), moe_ops.gated_act_ref(y[:, :N].float(), y[:, N:].float())) < BF16


@pytest.mark.parametrize("M", [129, 161, 300, 777])
@pytest.mark.parametrize("N,K", [(128, 1024), (136, 1024), (264, 1016), (392, 1088), (3848, 4096)])
def test_projections_of_prompts_on_pairs_of_ctas(M, N, K):
    """One row tile, a second tile that only one CTA of a pair has rows of, sums on either side of where pairs start; last token tiles of which a
    CTA's half is short."""
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(2 * N, K, device=DEV) * K ** -0.5).bfloat16()
    res = torch.randn(M, N, device=DEV).bfloat16()
    y = x.double() @ w.double().t()
    # products of bf16 are exact in fp32, and the sums are a thousandth of the result's rounding
    assert rel_l2(ops.linear(x, w[:N], residual=res), y[:, :N] + res.double()) < BF16
    assert rel_l2(ops.linear(x, w[:N], out_dtype=torch.float32), y[:, :N]) < BF16 / 256
    got, ssq = ops.linear(x, w[:N], residual=res, want_ssq=True)
    assert rel_l2(ssq.sum(-1), got.double().square().sum(-1)) < 1e-5
    assert rel_l2(ops.gated_linear(x, w, N), moe_ops.gated_act_ref(y[:, :N].float(), y[:, N:].float())) < BF16


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K,group,gated", [(4752, 3072, 64, False), (4736, 3072, 64, False), (4744, 5120, 128, False), (2 * 4736, 3136, 64, True),
                                             (2848, 8192, 64, False), (2848, 8448, 128, False), (2832, 8192, 64, False), (4752, 17600, 64, False), (2 * 2384, 17664, 64, True),
                                             (71040, 128, 64, False), (35520, 960, 64, False)])
@pytest.mark.parametrize("decades", [0, 6])
def test_four_bit_rows_on_integer_products(M, N, K, group, gated, decades):
    """On either side of where one or two tokens take the persistent kernel, with and without a split of K; row tiles that are no whole rounds,
    K blocks that leave warps without any; activations of one size and over six decades; rows that are part of wider ones."""
    ql = QuantLinear.from_dense((torch.randn(N, K, device=DEV) * 0.05).bfloat16(), 4, group)
    x = torch.randn(M, K + 8, device=DEV) * 10.0 ** (torch.rand(M, K + 8, device=DEV) * decades - decades / 2)
    x = x.bfloat16()[:, :K]
    y = x.double() @ ql.dequantize(torch.float32).double().t()
    res = torch.randn(M, N, device=DEV).bfloat16()
    ref = moe_ops.gated_act_ref(y[:, :N // 2].float(), y[:, N // 2:].float()) if gated else (y + res.double()).float()
    got = ql.gated(x) if gated else ql(x, residual=res)
    assert rel_l2(got, ref) < BF16
    if not gated:
        # fp32 results: a block's numbers are kept to 2^-21 of its largest, and 64 of them times at most 15 steps around zero are summed in fp32
        assert rel_l2(ql(x, out_dtype=torch.float32), y) < 2.0 ** -18
    x[0, K - 5] = float("inf")
    assert bool(torch.isnan(ql.gated(x) if gated else ql(x)).all(-1)[0]) and (M == 1 or bool(torch.isfinite(ql(x)[1]).all()))


@pytest.mark.parametrize("M,N,K,group,gated", [(1, 9488, 18624, 64, False), (1, 2 * 4752, 20608, 128, True), (2, 9488, 9408, 64, False),
                                               (2, 26000, 10624, 128, False), (2, 2 * 4752, 9280, 64, True), (2, 2 * 16400, 9344, 64, True)])
def test_four_bit_rows_over_many_rounds_of_two_ctas(M, N, K, group, gated):
    """Matrices of three and more rounds whose activations do not fit one CTA: the buffers and barriers of the exchange are used again."""
    ql = QuantLinear.from_dense((torch.randn(N, K, device=DEV) * 0.05).bfloat16(), 4, group)
    x = torch.randn(M, K, device=DEV).bfloat16()
    y = x.double() @ ql.dequantize(torch.float32).double().t()
    ref = moe_ops.gated_act_ref(y[:, :N // 2].float(), y[:, N // 2:].float()) if gated else y
    got = [ql.gated(x) if gated else ql(x, out_dtype=torch.float32) for _ in range(20)]
    assert rel_l2(got[0], ref) < (BF16 if gated else 2.0 ** -18)      # fp32 results as in test_four_bit_rows_on_integer_products
    assert all(torch.equal(g, got[0]) for g in got)


@pytest.mark.parametrize("M,K", [(512, 1024), (513, 1024), (2048, 1024), (2049, 1024), (2049, 2048), (513, 2112), (4001, 64)])
def test_gated_four_bit_prompts_of_short_sums(M, K):
    """On either side of where the activation has a kernel of its own."""
    ql = QuantLinear.from_dense((torch.randn(2 * 520, K, device=DEV) * 0.05).bfloat16(), 4, 64)
    x = torch.randn(M, K, device=DEV).bfloat16()
    y = x.double() @ ql.dequantize(torch.float32).double().t()
    # the kernel of its own reads gate and up rounded to bf16, and both forms multiply bf16 weights
    assert rel_l2(ql.gated(x), moe_ops.gated_act_ref(y[:, :520].float(), y[:, 520:].float())) < 3 * BF16


@pytest.mark.parametrize("T", [1, 2, 3, 5, 64])
@pytest.mark.parametrize("H,inter", [(256, 96), (2048, 768)])
def test_experts_of_few_tokens(T, H, inter):
    """Steps with fewer routes than the plan has room for items."""
    E, k = 64, 8
    x = torch.randn(T, H, device=DEV).bfloat16()
    gu = (torch.randn(E, 2 * inter, H, device=DEV) / H ** 0.5).bfloat16()
    dn = (torch.randn(E, H, inter, device=DEV) / inter ** 0.5).bfloat16()
    logits = torch.randn(T, E, device=DEV)
    ids, w, plan, xp = moe_ops.route_plan_gather(logits, x, k, "softmax", True, 1.0, None, 0, E)
    got = moe_ops.experts_forward(x, ids, w, gu, dn, plan=plan, xp=xp)
    # the product of gate and up and every expert's row are rounded to bf16 on both sides, the sum on this one
    assert rel_l2(got, moe_ops.experts_ref(x, ids, w, gu, dn)) < 2 * BF16


@pytest.mark.parametrize("D,n_q,n_kv", [(128, 32, 8), (64, 8, 8), (128, 16, 1), (64, 12, 2), (128, 32, 1)])
@pytest.mark.parametrize("q_lens,kv_lens,window,sinks", [
    ([45], [4141], 0, False),                       # the next message of a chat
    ([1, 5, 130], [2000, 77, 130], 0, True),        # beside each other: one that sees fewer tiles than there are splits
    ([16, 17, 64, 65], [1024, 1025, 639, 1153], 0, False),
    ([33, 2], [1500, 3000], 200, True),             # parts of the keys that no row of a cluster's CTA sees
    ([300, 7], [3000, 900], 0, False)])             # more than one tile of rows
def test_attention_of_short_portions(D, n_q, n_kv, q_lens, kv_lens, window, sinks):
    pages = [(n + 15) // 16 for n in kv_lens]
    kc, vc = (torch.randn(sum(pages) + 1, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
    bt = torch.zeros(len(pages), max(pages) + 3, dtype=torch.int32, device=DEV)
    ids, at = torch.randperm(sum(pages), device=DEV).int() + 1, 0
    for i, n in enumerate(pages):
        bt[i, :n] = ids[at:at + n]
        at += n
    q = (torch.randn(sum(q_lens), n_q, D, device=DEV) * 1.5).bfloat16()
    cu = torch.tensor([0] + torch.tensor(q_lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    lens = torch.tensor(kv_lens, dtype=torch.int32, device=DEV)
    sink = torch.randn(n_q, device=DEV) if sinks else None
    args = (q, kc, vc, bt, lens, cu, max(q_lens), D ** -0.5)
    got = ops.attention_prefill(*args, window=window, sinks=sink, max_kv_len=max(kv_lens))
    ref = ops.attention_ref(q, kc, vc, bt, lens, q_lens, D ** -0.5, window, sink)
    whole = ops.attention_prefill(*args, window=window, sinks=sink)       # unsplit, a query head per CTA
    # probabilities and the result are rounded to bf16; the two forms sum in another order
    assert rel_l2(got, ref) < 2 * BF16 and rel_l2(got, whole) < 2 * BF16
    # a context the host understates only changes the split
    assert rel_l2(ops.attention_prefill(*args, window=window, sinks=sink, max_kv_len=600), whole) < 2 * BF16


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(16, 8), (128, 2048), (144, 2056), (2048, 1000), (1040, 4096), (256, 6152)])
def test_rows_of_one_and_two_tokens(M, N, K):
    """Pieces of K that do not fill a pass of the CTA or its two batches, columns that do not fill a cluster; all of the epilogue."""
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    bias, res = torch.randn(N, device=DEV).bfloat16(), torch.randn(M, N, device=DEV).bfloat16()
    parts = torch.rand(M, 5, device=DEV) * K
    scale = torch.rsqrt(parts.sum(-1, keepdim=True) / K + 1e-5)
    ref = (x.float() @ w.float().t()) * scale + bias.float() + res.float()
    for split in (0, 1):          # 1: the tensor-core kernel
        y, ssq = ops.linear(x, w, bias=bias, residual=res, row_ssq=parts, norm_eps=1e-5, want_ssq=True, force_split=split)
        assert rel_l2(y, ref) < BF16 and ssq.shape == (M, (N + 127) // 128)
        want = torch.nn.functional.pad(y.float() ** 2, (0, -N % 128)).view(M, -1, 128).sum(-1)
        assert bool(((ssq - want).abs() <= 128 * 2.0 ** -24 * want + 1e-30).all())
    y = ops.linear(x, w, out_dtype=torch.float32, activation="relu2")
    assert rel_l2(y, torch.relu(x.float() @ w.float().t()) ** 2) < 1e-5


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(4736, 64), (4752, 64), (4144, 1016), (4160, 1016), (4736, 1024), (3552, 512), (3568, 512), (3072, 2048), (3088, 2048)])
def test_rows_of_one_and_two_tokens_at_the_borders_of_a_round(M, N, K):
    test_rows_of_one_and_two_tokens(M, N, K)


@pytest.mark.parametrize("M", [257, 2049, 2304, 4100])
def test_prompt_gemm_bands(M):
    """Token tiles that do not fill a band, and a last one that is nearly empty."""
    w, x = (torch.randn(1160, 192, device=DEV) / 14).bfloat16(), torch.randn(M, 192, device=DEV).bfloat16()
    assert rel_l2(ops.linear(x, w), x.float() @ w.float().t()) < BF16


@pytest.mark.parametrize("R,V", [(1, 128256), (1, 4097), (7, 32002), (33, 40000), (300, 1000)])
def test_largest_logit_over_a_cluster(R, V):
    from eredu_b200.ops.sampling import SamplingParams, pack_rows

    logits = torch.randn(R, V, device=DEV).round(decimals=1)           # many equal ones: the smallest token wins
    rows = torch.from_numpy(pack_rows([SamplingParams(temperature=0.0)] * R, [1] * R, hist_lens=[0] * R, stream_ids=[0] * R).view("u1").copy()).view(R, -1).to(DEV)
    allow = torch.rand(V, device=DEV) < 0.5
    mask = ops.pack_allow_mask(allow)
    for a, m in ((None, torch.ones_like(allow)), (mask[None], allow)):
        want = logits.masked_fill(~m, float("-inf"))
        want = (want == want.amax(-1, keepdim=True)).int().argmax(-1)
        probs = torch.full((R, V), 7.0, device=DEV)
        got = ops.sample(logits.clone(), rows, allow=a, probs=probs, all_greedy=True)
        assert torch.equal(got.long(), want) and torch.equal(probs.argmax(-1), want) and bool((probs.sum(-1) == 1).all())
    logits[0, V - 1] = 100.0
    assert int(ops.sample(logits, rows, all_greedy=True)[0]) == V - 1


@pytest.mark.parametrize("R,V", [(13, 48000), (14, 50257), (32, 24004), (33, 47999), (37, 48000), (74, 50000), (75, 50000), (2, 23996)])
def test_largest_logit_at_the_borders_of_the_rule(R, V):
    test_largest_logit_over_a_cluster(R, V)


@pytest.mark.parametrize("T,k,H", [(1, 8, 2048), (3, 1, 1000), (64, 6, 4104), (2, 32, 64)])
def test_weighted_expert_rows(T, k, H):
    """Slots that do not fill a batch, columns that do not fill a CTA, routes of other ranks; sums of squares of what is stored."""
    rows, w = torch.randn(T * k, H, device=DEV).bfloat16(), torch.rand(T, k, device=DEV)
    res, extra = torch.randn(T, H, device=DEV).bfloat16(), torch.randn(T, H, device=DEV).bfloat16()
    pos = torch.randperm(T * k, device=DEV).int()
    if k > 1:
        pos[1::5] = -1
    out, ssq = torch.empty_like(res), torch.empty(T, (H + 1023) // 1024, device=DEV)
    code = moe_ops.lib().eredu_moe_combine_ssq(*map(moe_ops.ptr, (rows, pos, w, res, extra, out, ssq)), T, k, H, moe_ops.stream_ptr(out.device))
    assert code == 0
    ref = res.float() + extra.float() + moe_ops.RoutedRows(rows, pos, w).summed()
    assert rel_l2(out, ref) < BF16
    assert torch.allclose(ssq.sum(-1), out.float().square().sum(-1), rtol=H * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("T,k,H", [(1023, 1, 1000), (1024, 1, 1000), (1500, 2, 4104), (1024, 3, 64)])
def test_weighted_expert_rows_of_prompts(T, k, H):
    """Few slots of many tokens have a kernel of their own; both add in one order."""
    rows, w = torch.randn(T * k, H, device=DEV).bfloat16(), torch.rand(T, k, device=DEV)
    res = torch.randn(T, H, device=DEV).bfloat16()
    pos = torch.randperm(T * k, device=DEV).int()
    pos[1::5] = -1
    out, other, ssq = torch.empty_like(res), torch.empty_like(res), torch.empty(T, (H + 1023) // 1024, device=DEV)
    p, stream = moe_ops.ptr, moe_ops.stream_ptr(out.device)
    assert moe_ops.lib().eredu_moe_combine(p(rows), p(pos), p(w), p(res), None, p(out), T, k, H, stream) == 0
    assert moe_ops.lib().eredu_moe_combine_ssq(p(rows), p(pos), p(w), p(res), None, p(other), p(ssq), T, k, H, stream) == 0
    assert torch.equal(out, other) and rel_l2(out, res.float() + moe_ops.RoutedRows(rows, pos, w).summed()) < BF16


@pytest.mark.parametrize("E,e0,e1,routes,k", [(128, 0, 128, 8192, 8), (8, 2, 6, 4096, 2), (512, 0, 512, 5000, 10), (60, 0, 30, 33, 3), (1, 0, 1, 40, 1)])
def test_expert_plan_keeps_the_order_of_the_routes(E, e0, e1, routes, k):
    ids = torch.randint(0, E, (routes // k, k), device=DEV, dtype=torch.int32)
    plan = moe_ops.ExpertPlan(ids, k, e0, e1, 64, ids.numel())
    flat = ids.flatten().cpu()
    order = [r for e in range(e0, e1) for r in (flat == e).nonzero().flatten().tolist()]
    want = torch.full((flat.numel(),), -1, dtype=torch.int32)
    want[order] = torch.arange(len(order), dtype=torch.int32)
    assert torch.equal(plan.route_pos.cpu(), want)
    assert torch.equal(plan.row_token[:len(order)].cpu(), torch.tensor(order, dtype=torch.int32) // k)
    assert plan.seg.tolist() == [int(((flat >= e0) & (flat < e0 + i)).sum()) for i in range(e1 - e0 + 1)]


@pytest.mark.parametrize("T,E,e0,n_local,k", [(1, 128, 0, 128, 8), (4, 128, 0, 128, 8), (5, 128, 0, 128, 8), (1, 512, 128, 256, 10), (3, 8, 2, 4, 2),
                                              (16, 4, 0, 4, 2), (17, 4, 0, 4, 1), (32, 64, 0, 64, 1), (1, 16, 12, 4, 1)])
def test_routes_of_few_tokens_are_planned_alike(T, E, e0, n_local, k):
    """Up to 32 routes, compared by the lanes of a warp, against the general plan of the same routes; experts elsewhere, and none at all."""
    logits, x = torch.randn(T, E, device=DEV), torch.randn(T, 256, device=DEV).bfloat16()
    if T == 1 and E == 16:
        logits[0, 3] = 9.0
    ids, _, plan, xp = moe_ops.route_plan_gather(logits, x, k, "softmax", True, 1.0, None, e0, n_local)
    want = moe_ops.ExpertPlan(ids, k, e0, e0 + n_local, plan.tile, T * k)
    rows = int(want.counts[0])
    assert torch.equal(plan.counts, want.counts) and torch.equal(plan.work, want.work) and torch.equal(plan.seg, want.seg)
    assert torch.equal(plan.route_pos, want.route_pos) and torch.equal(plan.row_token[:rows], want.row_token[:rows])
    assert torch.equal(xp[:rows], x[want.row_token[:rows].long()])


@pytest.mark.parametrize("T,k", [(16, 2), (10, 3), (9, 2), (1, 3)])
def test_routes_of_few_tokens_that_choose_an_expert_twice(T, k):
    """The one kept group holds one expert, so that the other routes of a token go to the first of what is left: more rows than an item has."""
    logits, x = torch.randn(T, 8, device=DEV), torch.randn(T, 256, device=DEV).bfloat16()
    logits[:, 0] = 9.0
    ids, _, plan, xp = moe_ops.route_plan_gather(logits, x, k, "softmax", True, 1.0, None, 0, 8, n_group=8, topk_group=1)
    want = moe_ops.ExpertPlan(ids, k, 0, 8, plan.tile, T * k)
    assert torch.equal(plan.counts, want.counts) and torch.equal(plan.work, want.work) and torch.equal(plan.seg, want.seg)
    assert torch.equal(plan.route_pos, want.route_pos) and torch.equal(plan.row_token, want.row_token)
    assert torch.equal(xp, x[want.row_token.long()])


@pytest.mark.parametrize("E,e0,e1,routes,k", [(8, 0, 8, 3000, 2), (9, 0, 9, 3000, 3), (20, 4, 20, 130, 2)])
def test_expert_plan_of_few_experts(E, e0, e1, routes, k):
    """On either side of where lanes find their like by values instead of bits; batches of routes that end early."""
    test_expert_plan_keeps_the_order_of_the_routes(E, e0, e1, routes, k)


@pytest.mark.parametrize("M", [1, 64, 65])
@pytest.mark.parametrize("H", [2048, 2056, 4104, 8192])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_of_few_wide_rows(M, H, residual):
    x, w = torch.randn(M, H, device=DEV).bfloat16(), torch.rand(H, device=DEV) + 0.5
    r = torch.randn(M, H, device=DEV).bfloat16() if residual else None
    y, h = ops.rmsnorm(x, w, 1e-5, residual=r, weight_offset=0.25)
    yr, hr = ops.rmsnorm_ref(x, w, 1e-5, r, 0.25)
    assert rel_l2(y, yr) < BF16 and (h is None if not residual else torch.equal(h, hr))


@pytest.mark.parametrize("M,N,K", [(1024, 128, 512), (300, 96, 320), (700, 60, 2048)])
def test_router_of_prompts(M, N, K):
    """A narrow fp32 output over many tokens: small token tiles."""
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    y = ops.linear(x, w, out_dtype=torch.float32)
    assert rel_l2(y, x.float() @ w.float().t()) < 1e-5


@pytest.mark.parametrize("M", [257, 300, 1024, 2048, 4099, 9000])
@pytest.mark.parametrize("N,K", [(128, 2048), (96, 320), (256, 4096)])
def test_router_sums_have_one_order(M, N, K):
    """Logits that decide between experts do not depend on how many tokens stand beside them: every tile size adds K in one order."""
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    y = ops.linear(x, w, out_dtype=torch.float32)
    alone = torch.cat([ops.linear(x[i:i + 128], w, out_dtype=torch.float32, force_split=1) for i in range(0, M, 128)])
    assert torch.equal(y, alone)


@pytest.mark.parametrize("M", [65, 96, 100, 128, 129])
@pytest.mark.parametrize("N,K", [(8, 4096), (128, 2048), (96, 320), (256, 4096), (9600, 1088)])
def test_router_sums_of_short_prompts_have_the_same_order(M, N, K):
    x, w = torch.randn(300, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    assert torch.equal(ops.linear(x[:M], w, out_dtype=torch.float32), ops.linear(x, w, out_dtype=torch.float32)[:M])


@pytest.mark.parametrize("M,N,K", [(130, 1096, 256), (400, 4736, 128), (1250, 4096, 192), (1900, 2048, 128)])
@pytest.mark.parametrize("gated", [False, True])
def test_prompt_gemm_tiles_of_fewer_tokens(M, N, K, gated):
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(2 * N if gated else N, K, device=DEV) / K ** 0.5).bfloat16()
    y = x.float() @ w.float().t()
    if gated:
        assert rel_l2(ops.gated_linear(x, w, N), moe_ops.gated_act_ref(y[:, :N], y[:, N:])) < BF16
    else:
        assert rel_l2(ops.linear(x, w), y) < BF16


@pytest.mark.parametrize("D,n_q,n_kv,new,lens", [(128, 32, 8, 1, [2040]), (64, 8, 8, 1, [15, 16, 17, 1, 640]), (128, 64, 2, 5, [33, 700])])
def test_decode_attention_ahead_of_its_projection(D, n_q, n_kv, new, lens):
    """Steps of projection, attention and output projection without a synchronisation between them, each reading what the step before has
    appended: pages fetched ahead of the projection give the same bits as pages fetched behind it."""
    B, width, hidden, steps = len(lens), (n_q + 2 * n_kv) * D, 512, 6
    pages = [(n + steps * new + 15) // 16 for n in lens]
    bt = torch.zeros(B, max(pages), dtype=torch.int32, device=DEV)
    ids, at = torch.randperm(sum(pages), device=DEV).int(), 0
    for i, n in enumerate(pages):
        bt[i, :n] = ids[at:at + n]
        at += n
    w = (torch.randn(width, hidden, device=DEV) / hidden ** 0.5).bfloat16()
    wo = (torch.randn(hidden, n_q * D, device=DEV) / (n_q * D) ** 0.5).bfloat16()
    start = [torch.randn(sum(pages), n_kv, 16, D, device=DEV).bfloat16() for _ in range(2)]
    x0 = torch.randn(B * new, hidden, device=DEV).bfloat16()
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device=DEV).float() / D))
    table, plan = bt.cpu().long(), []
    for s in range(steps):
        pos = torch.tensor([n + s * new + i for n in lens for i in range(new)])
        rows = torch.arange(B).repeat_interleave(new)
        plan.append((pos.int().to(DEV), (table[rows, pos // 16] * 16 + pos % 16).to(DEV), torch.tensor([n + (s + 1) * new for n in lens], dtype=torch.int32, device=DEV)))
    results = []
    for settled in (False, True):
        kc, vc = start[0].clone(), start[1].clone()
        torch.cuda.synchronize()
        x, outs = x0, []
        for pos, slots, seq in plan:
            qkv = ops.linear(x, w)
            a = ops.attention_decode_rope(qkv, kc, vc, bt, seq, new, D ** -0.5, pos, slots, inv, n_q, n_kv, D, splits=2, settled=settled)
            x = ops.linear(a.view(B * new, -1), wo)
            outs.append(x)
        results.append((torch.stack(outs), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("E,k,T,H,inter", [(8, 2, 100, 512, 1472), (8, 2, 108, 512, 1472), (8, 2, 512, 256, 192), (16, 4, 260, 256, 320),
                                           (48, 4, 48, 512, 1088), (48, 4, 148, 512, 1088), (48, 4, 180, 512, 1088), (64, 4, 420, 256, 128), (4, 2, 80, 512, 320),
                                           (4, 2, 82, 512, 320), (64, 4, 224, 256, 128), (64, 4, 225, 256, 128), (8, 2, 128, 512, 1472),
                                           (8, 2, 132, 512, 1472)])
def test_experts_at_the_borders_of_the_rule(E, k, T, H, inter):
    """Few experts with 25 to 128 rows each; experts whose rows fill one item of sixteen and such that need a second."""
    x = torch.randn(T, H, device=DEV).bfloat16()
    gu = (torch.randn(E, 2 * inter, H, device=DEV) / H ** 0.5).bfloat16()
    dn = (torch.randn(E, H, inter, device=DEV) / inter ** 0.5).bfloat16()
    ids, w = moe_ops.route(torch.randn(T, E, device=DEV), k, "softmax", True, 1.0, None, 1, 1)
    # the product of gate and up and every expert's row are rounded to bf16 on both sides, the sum on this one
    assert rel_l2(moe_ops.experts_forward(x, ids, w, gu, dn), moe_ops.experts_ref(x, ids, w, gu, dn)) < 2 * BF16


@pytest.mark.parametrize("D", [64, 128])
def test_what_is_no_number_stays_none_when_keys_are_split(D):
    """A query that is no number, and a cached key that is none: the rows that meet them, and no others."""
    n_q, n_kv, new, kv = 32, 8, 20, 2000
    pages = (kv + 15) // 16
    kc, vc = (torch.randn(pages, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
    bt = torch.arange(pages, device=DEV, dtype=torch.int32)[None]
    q = torch.randn(new, n_q, D, device=DEV).bfloat16()
    lens, cu = torch.tensor([kv], device=DEV, dtype=torch.int32), torch.tensor([0, new], device=DEV, dtype=torch.int32)
    clean = ops.attention_prefill(q, kc, vc, bt, lens, cu, new, D ** -0.5, max_kv_len=kv)
    q[7, 3] = float("nan")
    kc[(kv - 5) // 16, 6, (kv - 5) % 16] = float("nan")       # seen by the last five tokens, heads 24 to 27
    want = torch.zeros(new, n_q, dtype=torch.bool, device=DEV)
    want[7, 3] = True
    want[new - 5:, 24:28] = True
    for split in (0, kv):
        got = ops.attention_prefill(q, kc, vc, bt, lens, cu, new, D ** -0.5, max_kv_len=split)
        assert torch.equal(got.isnan().any(-1), want) and torch.equal(got.isnan().all(-1), want)
        assert not split or torch.equal(got[~want], clean[~want])


@pytest.mark.parametrize("V", [32002, 128256])
def test_largest_logit_among_what_is_none(V):
    """Whole parts of a row that are masked, minus infinity or no number, and a row of nothing else."""
    from eredu_b200.ops.sampling import SamplingParams, pack_rows

    inf, nan = float("inf"), float("nan")
    logits = torch.randn(6, V, device=DEV)
    logits[0, :V - 10] = -inf
    logits[1, 10:] = nan
    logits[2] = -inf
    logits[3] = nan
    logits[4, V // 3] = inf
    allow = torch.ones(6, V, dtype=torch.bool, device=DEV)
    allow[5, :V - 100] = False
    rows = torch.from_numpy(pack_rows([SamplingParams(temperature=0.0)] * 6, [1] * 6, hist_lens=[0] * 6, stream_ids=[0] * 6).view("u1").copy()).view(6, -1).to(DEV)
    masks = torch.stack([ops.pack_allow_mask(a) for a in allow])
    want = logits.masked_fill(~allow | logits.isnan(), -inf).argmax(-1)
    want[2:4] = 0                                              # nothing is larger than the start of the search
    assert torch.equal(ops.sample(logits.clone(), rows, allow=masks, all_greedy=True).long(), want)


@pytest.mark.parametrize("new", [64, 65])
@pytest.mark.parametrize("kv", [1024 + 65, 4096 + 65])
def test_short_portions_on_either_side_of_a_cluster(new, kv):
    """Three portions of heads in groups of eight: 24 tiles of rows, which four CTAs share, and 36, for which clusters of four have no room."""
    n_q, n_kv, D, B = 32, 4, 128, 3
    pages = (kv + 15) // 16
    kc, vc = (torch.randn(B * pages, n_kv, 16, D, device=DEV).bfloat16() for _ in range(2))
    bt = torch.randperm(B * pages, device=DEV).int().view(B, pages)
    q = torch.randn(B * new, n_q, D, device=DEV).bfloat16()
    lens, cu = torch.full((B,), kv, device=DEV, dtype=torch.int32), torch.arange(B + 1, device=DEV, dtype=torch.int32) * new
    whole = ops.attention_prefill(q, kc, vc, bt, lens, cu, new, D ** -0.5)
    # probabilities are rounded to bf16 in front of the second product on both sides, against different maxima, and outputs once more
    assert rel_l2(ops.attention_prefill(q, kc, vc, bt, lens, cu, new, D ** -0.5, max_kv_len=kv), whole) < 2 * BF16
