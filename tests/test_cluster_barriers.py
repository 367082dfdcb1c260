"""Stores into the shared memory of another CTA: the CTAs of a cluster are placed together, but only a cluster barrier says that they run."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "eredu_b200" / "csrc" / "kernels"


# what reaches into another CTA: stores by their instruction, and calls of the helpers around st.async, remote arrivals and copies that count there
REMOTE = re.compile(r"st\.shared::cluster|(?<!void )\b(st_async\w*|store_async|mbar_arrive_cluster|tma_load_2d_pair_hint|umma_commit_pair)\(")
HELPERS = re.compile(r"__device__ __forceinline__ void (\w+)\([^{]*\{[^}]*?(?:st\.async|mbarrier\.arrive\.shared::cluster|\.cta_group::2\.L2|multicast::cluster)")


def unguarded_stores(source):
    """Lines of remote accesses that no wait on the cluster barrier dominates: a wait counts while the block that it stands in is open."""
    found, depth, waits = [], 0, []
    for number, line in enumerate(source.splitlines(), 1):
        code = re.sub(r"//.*", "", line)
        if REMOTE.search(code) and not waits:
            found.append(number)
        code = re.sub(r'"[^"]*"', '""', code)
        for token in re.findall(r"[{}]|cluster_wait_acquire\(\)", code):
            if token == "{":
                depth += 1
            elif token == "}":
                depth -= 1
                waits = [d for d in waits if d <= depth]
            else:
                waits.append(depth)
    assert depth == 0
    return found


@pytest.mark.parametrize("text, lines", [
    ("void f() {\n cluster_wait_acquire();\n if (a) {\n  asm(\"st.shared::cluster.f32 [%0], {%1};\");\n }\n}", []),
    ("void f() {\n if (a) {\n  cluster_wait_acquire();\n }\n asm(\"st.shared::cluster.f32\");\n}", [5]),
    ("void f() {\n cluster_wait_acquire();\n}\nvoid g() {\n asm(\"st.shared::cluster.f32\");\n}", [5]),
    ("void st_async(uint32_t a) {\n asm(\"st.async.weak\");\n}\nvoid f() {\n st_async(a);\n cluster_wait_acquire();\n st_async(b);\n}", [5]),
    ("void f() {\n store_async(a, v, b);\n st_async_f32(a, v, b);\n mbar_arrive_cluster(b);\n umma_commit_pair(b);\n}", [2, 3, 4, 5]),
    ("void f() {\n if (PAIR) cluster_wait_acquire();\n if (PAIR) tma_load_2d_pair_hint(a);\n}", [])])
def test_reading_of_blocks(text, lines):
    assert unguarded_stores(text) == lines


def test_helpers_of_remote_accesses_are_known():
    """A helper around one of these instructions is looked for by its name."""
    sources = sorted(KERNELS.glob("*.cu*")) + [KERNELS.parent / "common" / "ptx.cuh"]
    names = {name for path in sources for name in HELPERS.findall(path.read_text())}
    assert len(names) >= 6 and all(REMOTE.search(f" {name}(") for name in names), names


@pytest.mark.parametrize("name", sorted(p.name for p in KERNELS.glob("*.cu*")))
def test_remote_stores_wait_for_their_target(name):
    assert unguarded_stores((KERNELS / name).read_text()) == []


def round_of(source):
    """Reads, barriers and sends of a round of the persistent 4-bit kernel, in the order of the source."""
    loop = source[source.index("for (int r = 0; r < rounds; ++r)"):source.index("finish_exchange(rounds - 1)")]
    return re.findall(r"finish_exchange|__syncthreads|store_async|recv\[", re.sub(r"//.*", "", loop))


def test_sums_are_sent_behind_the_reads_of_the_round_before():
    """A CTA sends behind a barrier that follows its reads of the round before, so that who has its sums may write over what it has read. Its own
    sums take the same way: a plain store would need a barrier between itself and the reads as well."""
    assert round_of((KERNELS / "qgemv_stream.cu").read_text()) == ["finish_exchange", "__syncthreads", "store_async"]


def silent_decisions(source):
    """Lines that go by the outcome of a wait without a status word."""
    return [number for number, line in enumerate(source.splitlines(), 1)
            if re.search(r"mbar_wait\w*\([^;]*, nullptr, 0\)", line) and not re.search(r"^\s*(for \([^;]*;[^;]*;[^;]*\) )?mbar_wait\w*\(", line)]


@pytest.mark.parametrize("text, lines", [("  for (int i = 0; i < n; ++i) mbar_wait(&full[i], 0, nullptr, 0);\n  mbar_wait(&bars[i], parity, nullptr, 0);", []),
                                         ("const bool all = mbar_wait(&sent, 0, nullptr, 0);", [1]), ("if (!mbar_wait(&sent, 0, nullptr, 0)) return;", [1])])
def test_reading_of_waits(text, lines):
    assert silent_decisions(text) == lines


@pytest.mark.parametrize("name", sorted(p.name for p in KERNELS.glob("*.cu*")))
def test_waits_that_run_out_say_so(name):
    """Results that a wait decides on are missing when it runs out; only copies on their way out of a kernel are waited for without a word."""
    assert silent_decisions((KERNELS / name).read_text()) == []


def test_status_codes_have_names():
    codes = re.findall(r"kStatus\w+ = (\d+)", (KERNELS.parent / "common" / "ptx.cuh").read_text())
    from eredu_b200.ops.native import STATUS_NAMES
    assert sorted(map(int, codes)) == sorted(STATUS_NAMES)
