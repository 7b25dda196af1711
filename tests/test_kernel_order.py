"""Memory order that lockstep hardware would let go unnoticed, checked in the
kernels' sources: where lanes of a warp read what others stored, a __syncwarp
stands between (shuffles and ballots order no memory)."""
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(ROOT, "vehicleroutingproblem_b200", "csrc", "cuda")


def _function(file, name):
    """Text of the function `name`, comments removed."""
    with open(os.path.join(CUDA, file)) as f:
        lines = [line.split("//")[0] for line in f]
    text = "".join(lines)
    start = text.index(f" {name}(")
    at = text.index("{", start)
    depth, end = 1, at + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end]


def _between(text, first, last):
    a = text.index(first) + len(first)
    return text[a:text.index(last, a)]


def test_batch_fallback_reads_marked_elements_after_a_warp_barrier():
    build = _function("aco_batch.cu", "build_ants")
    for reader in ("coop_tier<", "coop_scan<"):
        assert "__syncwarp()" in _between(build, "if (none) {", reader)
    assert "__syncwarp()" in _between(build, "} while (none);", "us.mark(")


def test_batch_cost_reads_routes_after_a_warp_barrier():
    build = _function("aco_batch.cu", "build_ants")
    stores_to_loads = _between(build, "route[(pos & ~(LPA - 1)) + l] = held;", "load_nodes(0)")
    unconditional = stores_to_loads.split("if (rm)")[0]
    assert "__syncwarp()" in unconditional
    assert "__syncwarp()" in _between(stores_to_loads, "left -= added;", "} while (rm);")
