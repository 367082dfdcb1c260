"""Rules that choose how a launch is spread over the machine, as far as they are numbers."""
import pytest

from eredu_b200 import ops
from eredu_b200.ops import moe, native


@pytest.mark.parametrize("sms", [132, 148, 160])
@pytest.mark.parametrize("vocab", [8192, 32000, 50257, 128256, 262144])
def test_ctas_of_a_sampled_row_run_at_once(sms, vocab):
    """A CTA has 1024 threads with 63 registers: one fits an SM."""
    picks = [native.lib().eredu_sample_row_ctas(rows, vocab, sms) for rows in range(1, 300)]
    assert all(c == 1 or rows * c <= sms for rows, c in enumerate(picks, 1))
    assert picks == sorted(picks, reverse=True) and set(picks) <= {1, 2, 4, 8}
    assert picks[0] == (1 if vocab < 24000 else 4 if vocab < 48000 else 8)


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("ctas", [1, 2, 4, 8, 16, 24, 80])
def test_long_contexts_do_not_leave_most_of_the_gpu_idle(ctas, head_dim):
    """One CTA to an SM and eight to a cluster is the best plan of short contexts only: from some length on decode attention is split like that of a
    caller who knows nothing about the kernel, and stays so."""
    plan = lambda tokens: ops.decode_splits(ctas, 1, tokens, 148, rows=4, head_dim=head_dim)
    assert plan(512) <= ops.CLUSTER_SPLITS and plan(512) * ctas <= 148
    for tokens in (32768, 65536, 131072):
        assert plan(tokens) == ops.decode_splits(ctas, 1, tokens, 148)


@pytest.mark.parametrize("experts, inter", [(8, 14336), (16, 2048), (32, 512), (48, 768)])
def test_items_of_few_experts_leave_room_for_uneven_routes(experts, inter):
    """With 27 rows an expert on average, some have more than the 32 of a small item."""
    assert moe.expert_tile(26 * experts, experts, inter, 2048, True) == 32
    assert all(moe.expert_tile(rows * experts, experts, inter, 2048, True) == 256 for rows in range(27, 34))
