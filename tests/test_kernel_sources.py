"""What the kernels' sources must hold and no run can show: orderings whose loss is a rare race on shared memory."""
import glob
import os
import re

import pytest

import helpers

SOURCES = sorted(glob.glob(os.path.join(helpers.ROOT, "boring-llm_b200", "csrc", "*.cu*")))


def code(path):
    """The source without comments."""
    with open(path) as f:
        text = re.sub(r"/\*.*?\*/", " ", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_cluster_barriers_order_what_came_before(path):
    """A block that leaves behind a cluster barrier gives its shared memory to the next block. Whatever its peers sent there
    (arrivals on its barriers, partial sums) must be ordered before that: an arrival at a cluster barrier releases (the default,
    when no qualifier is given), or every arrival of a peer has been waited for. Only the product on pairs of SMs takes the second
    way, and only where no wait gave up."""
    text = code(path)
    relaxed = len(re.findall(r"barrier\.cluster\.arrive\.relaxed", text))
    if os.path.basename(path) != "gemm_tcgen05_pair.cu":
        assert relaxed == 0
        return
    guarded = re.findall(r"if \(\*give_up\) cluster_sync\(\);\s*else asm volatile\(\"barrier\.cluster\.arrive\.relaxed", text)
    assert relaxed == len(guarded)
    sent = re.findall(r"if \(([^;{}]*)\) mbar_arrive_leader\(acc_empty0", text)
    assert sent and len(sent) == len(re.findall(r"mbar_arrive_leader\(acc_empty0", text))
    assert all("t + 2 * n_pairs < total_tiles" in condition for condition in sent)
    assert re.search(r"for \(int j = max\(0, it - STAGES\); j < it; \+\+j\)\s*if \(!mbar_wait\(empty0", text)


@pytest.mark.parametrize("n_pairs", [1, 2, 3, 74])
@pytest.mark.parametrize("stages", [3, 5])
def test_every_arrival_in_the_product_on_pairs_is_waited_for(n_pairs, stages):
    """The loops of the kernel's loader, issuer and epilogue restated: for any number of tiles and k steps, the arrivals on
    acc_empty are those that the issuer waits for, and the commits on empty those that the loader waits for, phase by phase."""
    for total in list(range(1, 3 * n_pairs + 3)) + [5 * n_pairs, 7 * n_pairs + 1]:
        for pair in range(min(n_pairs, total)):
            tiles = range(pair, total, n_pairs)
            sent = [local for local, t in enumerate(tiles) if t + 2 * n_pairs < total]
            waited = [local - 2 for local, t in enumerate(tiles) if local >= 2]
            assert sent == waited
            for local in waited:                       # use n of a buffer waits for the phase of use n - 1
                assert (((local + 2) // 2) & 1) ^ 1 == (local // 2) & 1
            for steps in (1, 2, stages, stages + 1, 14):
                it = len(tiles) * steps
                refills = [(i - stages, ((i // stages) & 1) ^ 1) for i in range(stages, it)]
                tail = [(j, (j // stages) & 1) for j in range(max(0, it - stages), it)]
                assert [w for w, _ in refills + tail] == list(range(it))
                assert all(parity == (w // stages) & 1 for w, parity in refills + tail)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_warps_meet_before_they_take_or_free_tensor_memory(path):
    """tcgen05.alloc and dealloc are for a whole warp at once: behind code of one thread (setting up barriers, first copies) the
    warp's lanes meet before them."""
    text = code(path)
    for at in [m.start() for m in re.finditer(r"tcgen05\.(?:de)?alloc\b", text)]:
        before = text[:at]
        alone = max(before.rfind(s) for s in ("threadIdx.x == 0", "lane == 0", "elect_one()"))
        assert alone >= 0 and re.search(r"__syncwarp\(\)|__syncthreads\(\)", before[alone:])
