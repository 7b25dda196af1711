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


def test_bitmap_words_are_rewritten_after_a_warp_barrier():
    """Every lane of an ant writes the word back: one step's writes must not
    follow the next one's."""
    build = _function("aco_batch.cu", "build_ants")
    step = _between(build, "} while (none);", "us.mark(take ? next : 0)")
    assert "if (kBits) __syncwarp();" in step
    single = _function("aco_kernels.cu", "build_ant")
    assert "if (E != 1) __syncwarp();" in _between(single, "if (first == 0u) break;", "take_step(next")


def test_batch_cost_reads_routes_after_a_warp_barrier():
    build = _function("aco_batch.cu", "build_ants")
    stores_to_loads = _between(build, "route[(pos & ~(LPA - 1)) + l] = held;", "load_nodes(0)")
    unconditional = stores_to_loads.split("if (rm)")[0]
    assert "__syncwarp()" in unconditional
    assert "__syncwarp()" in _between(stores_to_loads, "left -= added;", "} while (rm);")


def test_construction_reads_the_epochs_weights_coherently():
    """The construction's blocks start while k_weights still writes the
    epoch's tables; the read-only path (__ldg) is for what no epoch writes."""
    with open(os.path.join(CUDA, "aco_kernels.cu")) as f:
        text = "".join(line.split("//")[0] for line in f)
    weight = _between(text, "uint32_t weight(uint32_t nb) const {", "}")
    assert "w[nb * step]" in weight and "__ldg" not in weight
    build = _function("aco_kernels.cu", "build_ant") + _function("aco_kernels.cu", "k_construct")
    for written in ("et.w", "et.rel", "et.rdep"):
        assert written in build and f"__ldg(a.{written}" not in build
