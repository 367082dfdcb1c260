"""Reads ahead of a kernel's dependency wait that are right only where every kernel releases the next one behind its own wait."""
import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parents[1] / "eredu_b200" / "csrc" / "kernels"


def test_lengths_and_pages_are_not_read_ahead_in_builds_that_release_at_entry():
    decode = (KERNELS / "attention.cu").read_text()
    writes = re.findall(r"p\.settled = ([^;]*);", decode)
    launches = [w for w in writes if "t0" in w]          # what the kernel sees; the entry point's flag only passes through it
    assert launches and all("!EREDU_PDL_EARLY &&" in w for w in launches)
    assert "settled = p.settled != 0" in decode and decode.count("settled = p.settled") == 2
    latent = (KERNELS / "latent_attention.cu").read_text()
    assert "if (EREDU_PDL_EARLY) pdl_wait();" in latent


def test_norm_weights_are_read_behind_the_wait():
    """They may be what the kernel just in front has written (a vector of ones, a converted weight)."""
    source = (KERNELS / "norm_rope.cu").read_text()
    kernel = source[source.index("rmsnorm_kernel(const"):]
    ahead = kernel[:kernel.index("pdl_wait();")]
    assert not re.search(r"\(w\)\[|= w\[", ahead)


def test_what_decode_attention_reads_ahead_is_promised_by_its_caller():
    """Everything that the kernel reads in front of its wait when its surroundings are settled is named where callers say that they are."""
    from eredu_b200 import ops
    source = (KERNELS / "attention.cu").read_text()
    kernel = source[source.index("attn_decode_kernel(AttnParams p) {"):]
    ahead = kernel[:kernel.index("if (settled) {")]
    arrays = set(re.findall(r"p\.(block_table|seq_lens|positions|slots|q_norm_w|k_norm_w|sinks)\b", ahead)) | ({"inv_freq"} if "turn_at" in ahead else set())
    promise = ops.attention_decode_rope.__doc__.partition("``settled``")[2]
    assert {"positions", "slots"} <= arrays and all(f"``{name}``" in promise for name in arrays), arrays
