"""Rules that choose how a launch is spread over the machine, as far as they are numbers."""
import pytest

from eredu_b200.ops import native


@pytest.mark.parametrize("sms", [132, 148, 160])
@pytest.mark.parametrize("vocab", [8192, 32000, 50257, 128256, 262144])
def test_ctas_of_a_sampled_row_run_at_once(sms, vocab):
    """A CTA has 1024 threads with 63 registers: one fits an SM."""
    picks = [native.lib().eredu_sample_row_ctas(rows, vocab, sms) for rows in range(1, 300)]
    assert all(c == 1 or rows * c <= sms for rows, c in enumerate(picks, 1))
    assert picks == sorted(picks, reverse=True) and set(picks) <= {1, 2, 4, 8}
    assert picks[0] == (1 if vocab < 24000 else 4 if vocab < 48000 else 8)
