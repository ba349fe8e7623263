"""Order of the barrier waits in the decode warps of the weight-decoding GEMM (csrc/kernels/gemm_wdec_kernel.cuh), on a model of
its rings: copies land in any order, and a parity wait passes whenever the phase has the other parity."""
import random
from pathlib import Path

import pytest

import deepseek_v4_2080ti_b200

SOURCE = Path(deepseek_v4_2080ti_b200.__file__).parent / "csrc" / "kernels" / "gemm_wdec_kernel.cuh"


def _kernel_order():
    """The two waits of a decode group in the order in which the kernel takes them."""
    text = SOURCE.read_text()
    body = text[text.index("if ((int)(it % G) != grp) continue;"):text.index("const uint8_t* raw = sRaw")]
    return sorted(("empty", "tma_full"), key=lambda name: body.index(f"mbar_wait(&{name}["))


def _stale_reads(order, groups, stages, blocks, seed):
    """K-blocks that a decode group unpacked from a raw stage which did not hold them.  Every role takes one step at a time, in
    an order drawn at random; a copy, once asked for, lands at a random later time."""
    rng = random.Random(seed)
    landed, committed = [0] * stages, [0] * stages           # completed phases of tma_full and empty
    decoded, holds = [0] * groups, [None] * stages
    asked = product = 0
    flying, at, step = [], list(range(groups)), [0] * groups      # a group's k-block, how many of its waits are over
    slow, stale = set(rng.sample(range(blocks), blocks // 6)), []
    passes = lambda phases, index: (phases & 1) != (index & 1)
    for _ in range(200 * blocks):
        if product == blocks:
            break
        role = rng.randrange(3 + groups)
        if role == 0 and asked < blocks and (asked < stages or passes(committed[asked % stages], asked // stages + 1)):
            flying.append(asked)
            asked += 1
        elif role == 1 and flying:
            it = flying[rng.randrange(len(flying))]
            if it in slow and rng.random() < 0.97:
                continue
            flying.remove(it)
            holds[it % stages] = it
            landed[it % stages] += 1
        elif role == 2 and product < blocks:
            it = product
            if passes(landed[it % stages], it // stages) and passes(decoded[it % groups], it // groups):
                committed[it % stages] += 1
                product += 1
        elif role >= 3:
            g = role - 3
            it = at[g]
            if it >= blocks:
                continue
            if step[g] < 2:
                if order[step[g]] == "tma_full":
                    step[g] += passes(landed[it % stages], it // stages)
                else:
                    prev = it - groups
                    step[g] += prev < 0 or passes(committed[prev % stages], prev // stages)
            else:
                if holds[it % stages] != it:
                    stale.append(it)
                decoded[g] += 1
                at[g], step[g] = it + groups, 0
    assert product == blocks
    return stale


# (decoded slots, raw stages): rings as deep as their slots, between one and two times as deep, and deeper
RINGS = [(4, 4), (4, 5), (4, 6), (4, 7), (4, 8), (4, 16), (6, 9), (6, 10), (8, 8), (8, 10), (8, 11), (8, 13), (8, 15)]


@pytest.mark.parametrize("groups,stages", RINGS)
def test_decode_warps_read_the_block_they_waited_for(groups, stages):
    order = _kernel_order()
    for seed in range(25):
        assert not _stale_reads(order, groups, stages, 150, seed)


def test_the_model_sees_the_race_of_the_other_order():
    assert any(_stale_reads(["tma_full", "empty"], 8, 11, 150, seed) for seed in range(25))
