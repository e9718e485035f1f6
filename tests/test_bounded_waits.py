"""Waits that run out, read from the sources (no GPU is made to wait for something that never comes): lanes of a warp that works
together give up together, and a block stays until the copies it asked for must have landed."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "burn_transformers_b200" / "csrc"
WAIT = re.compile(r"\b(?:tc_bar_wait|ta_bar_wait|lm_wait)\(")
ONE_LANE = ("tc_elect()", "ta_elect()", "lane == 0")
FILES = [p.name for p in sorted(CSRC.glob("*.cu")) if WAIT.search(p.read_text())]


def branches(lines, at):
    """The headers of the blocks around line `at`, by indentation, innermost first."""
    depth = len(lines[at]) - len(lines[at].lstrip())
    for line in reversed(lines[:at]):
        here = len(line) - len(line.lstrip())
        if line.strip() and not line.startswith("#") and here < depth:
            depth = here
            yield line
            if here == 0:
                return


@pytest.mark.parametrize("name", FILES)
def test_a_warp_gives_up_as_a_whole(name):
    lines = [re.sub(r"//.*", "", line) for line in (CSRC / name).read_text().split("\n")]
    for at, line in enumerate(lines):
        if not WAIT.search(line) or "__device__" in line:
            continue
        # a wait whose end a lane leaves its loop or branch for: in one lane alone, or by the vote of all
        leaves = "if (!" in line or (re.search(r"(const )?bool \w+ = ", line) and "if (!" in lines[at + 1])
        jumps = any(word in " ".join(lines[at:at + 5]) for word in ("break;", "return false;"))
        if leaves and jumps and "__all_sync" not in line:
            assert any(one in header for header in branches(lines, at) for one in ONE_LANE), f"{name}:{at + 1}: {line.strip()}"


@pytest.mark.parametrize("name", FILES)
def test_a_block_that_gives_up_stays_for_its_copies(name):
    for kernel in (CSRC / name).read_text().split("__global__")[1:]:
        kernel = kernel.split("\n}\n")[0]
        if WAIT.search(kernel):
            after = kernel[max(m.end() for m in WAIT.finditer(kernel)):]
            assert re.search(r"__syncthreads\(\);\s+if \(\*?failed\) let_copies_land\(\);", after), name
