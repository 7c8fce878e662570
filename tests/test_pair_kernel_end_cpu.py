"""The end of the pair GEMM, whose closing cluster barrier orders no memory: whatever one CTA sends to a barrier in the other's
shared memory has been waited for by then.  Read from the source and walked through on the CPU."""
import pathlib
import re

import pytest

SRC = (pathlib.Path(__file__).resolve().parent.parent / "csrc/gemm/gemm2_bf16.cu").read_text()
KERNEL = SRC[SRC.index("gemm2_bf16_kernel("):SRC.index("static int make_tmap_mn3d")]


def section(title):
    """The part of the kernel under this heading."""
    rest = KERNEL[KERNEL.index(title) + len(title):]
    return rest[:re.search(r"// -{20,}", rest[rest.index("\n"):]).start() + rest.index("\n")]


def test_the_issuer_waits_for_the_last_release_of_the_accumulators():
    issuer = section("MMA issuer (leader CTA only)")
    behind = issuer[issuer.rindex("umma_commit_pair(&tmem_full[buf])"):]
    assert re.search(r"for \(int i = 0; i < 2 && ok; \+\+i, \+\+local\)\s*"
                     r"ok = mbar_wait_warp\(&tmem_empty\[local & 1\], \(uint32_t\(local >> 1\) & 1\) \^ 1, ", behind)
    # every way out of the loop over tiles is either its end or a wait that ran out (whose warp must not wait again)
    assert not re.search(r"\)\)\s*break;", issuer) and issuer.count("ok = false; break;") == 1
    # and the barrier behind may stay relaxed only with that wait ahead of it
    assert KERNEL.index("MMA issuer") < KERNEL.index("barrier.cluster.arrive.relaxed")


class Barrier:
    """An mbarrier of `count` arrivals: the phase in progress; a wait for a parity is over once the phase of that parity is."""
    def __init__(self, count):
        self.count, self.arrived, self.phase = count, 0, 0

    def arrive(self):
        self.arrived += 1
        if self.arrived == self.count:
            self.arrived, self.phase = 0, self.phase + 1

    def passed(self, parity):
        return (self.phase & 1) != parity


@pytest.mark.parametrize("tiles", range(9))
@pytest.mark.parametrize("arrivals", [8, 16])
def test_those_waits_end_exactly_when_every_arrival_has_landed(tiles, arrivals):
    """The issuer runs ahead of the epilogue as far as its waits let it; the two waits behind its last tile do not end before
    the last of all arrivals, and do end then, for any number of tiles."""
    bars, owed, landed = [Barrier(arrivals), Barrier(arrivals)], [], 0

    def wait(local):
        nonlocal landed
        while not bars[local & 1].passed(((local >> 1) & 1) ^ 1):
            assert owed, "a wait that nothing ends"
            bars[owed.pop(0)].arrive()
            landed += 1

    for local in range(tiles):
        wait(local)
        owed += [local & 1] * arrivals
    for local in (tiles, tiles + 1):
        wait(local)
    assert landed == tiles * arrivals and not owed


def test_the_producers_wait_for_the_last_release_of_the_stages():
    producer = section("TMA producer (both CTAs)")
    behind = producer[producer.index("tma_load_2d_pair(sb + j"):]
    assert re.search(r"for \(int i = 0; i < STAGES && ok; \+\+i\) \{\s*"
                     r"ok = mbar_wait_warp\(&empty\[stage\], phase \^ 1, [^;]*;\s*"
                     r"if \(\+\+stage == STAGES\) \{ stage = 0; phase \^= 1; \}\s*\}", behind)


@pytest.mark.parametrize("stages", [5, 6, 8])
@pytest.mark.parametrize("blocks", [0, 1, 4, 5, 6, 7, 8, 13, 16, 24])
def test_those_waits_end_exactly_when_every_commit_has_landed(stages, blocks):
    bars, owed, landed = [Barrier(1) for _ in range(stages)], [], 0
    stage = phase = 0

    def step(load):
        nonlocal stage, phase, landed
        while not bars[stage].passed(phase ^ 1):
            assert owed, "a wait that nothing ends"
            bars[owed.pop(0)].arrive()
            landed += 1
        if load:
            owed.append(stage)
        stage += 1
        if stage == stages:
            stage, phase = 0, phase ^ 1

    for _ in range(blocks):
        step(True)
    for _ in range(stages):
        step(False)
    assert landed == blocks and not owed
