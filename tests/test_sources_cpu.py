"""Rules of the device sources that a run cannot show to be kept."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cp-paw_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return [re.sub(r"//.*", "", line) for line in f]


@pytest.mark.parametrize("name", SOURCES)
def test_warp_wide_instructions_are_volatile(name):
    """An .aligned instruction needs the whole warp: its asm statement is volatile,
    so that the compiler does not move it into code that only some lanes run."""
    text = "".join(code(name))
    for m in re.finditer(r"\basm\b(\s+volatile)?\s*\(", text):
        body = text[m.end():text.index(";", text.index(":", m.end()))] if ":" in text[m.end():] else text[m.end():]
        assert m.group(1) or ".aligned" not in body, f"{name}: {body[:60]!r}"


@pytest.mark.parametrize("name", SOURCES)
def test_products_start_with_a_converged_warp(name):
    """Every block of dmma calls follows a __syncwarp, with no conditional load from
    global memory between them."""
    lines = code(name)
    for at, line in enumerate(lines):
        if not re.search(r"\bdmma\(", line) or "__device__" in line:
            continue
        for back in range(at - 1, -1, -1):
            assert not re.search(r"^}|__ldcg|\? \*reinterpret_cast", lines[back]), f"{name}:{at + 1}: no __syncwarp"
            if "__syncwarp();" in lines[back]:
                break


@pytest.mark.parametrize("name", SOURCES)
def test_blocks_are_counted_after_every_threads_stores(name):
    """A block that counts itself as done for the launch's last block: every storing
    thread fences its stores, and a barrier stands between those fences and the
    count, which one thread makes for all of them."""
    lines = code(name)
    for at, line in enumerate(lines):
        if "atomicAdd(" not in line:
            continue
        barrier = fence = None
        for back in range(at - 1, -1, -1):
            if re.search(r"__sync(warp|threads)\(\)", lines[back]):
                barrier = back
            if "__threadfence();" in lines[back]:
                fence = back
                break
        assert fence is not None and barrier is not None and fence < barrier, f"{name}:{at + 1}"
