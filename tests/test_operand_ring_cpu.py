"""The barrier protocol of the swapped tile family's operand ring, played on the CPU with the scale warp's period from
csrc/dg_ring.cuh.  A breach of it shows on a GPU only by chance, and then as a launch failure."""
import ctypes
import os
import random
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgemm_rust_b200", "csrc")


def most_stages():
    with open(os.path.join(CSRC, "dg_gemm_kernel.cuh")) as f:
        return int(re.search(r"kMaxStages = (\d+)", f.read()).group(1))


@pytest.fixture(scope="module")
def scale_period(tmp_path_factory):
    path = tmp_path_factory.mktemp("ring")
    source, lib = path / "ring.cpp", path / "ring.so"
    source.write_text('#include "dg_ring.cuh"\nextern "C" uint32_t visit(uint32_t s, uint32_t p) { return dg::scale_period(s, p); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(source), "-o", str(lib)])
    return ctypes.CDLL(str(lib)).visit


class Barrier:
    """An mbarrier: a phase ends with its `count`-th arrival, a wait knows the parity of the phase it asks for."""

    def __init__(self, count):
        self.count, self.arrivals, self.phase = count, [], 0

    def arrive(self, tag):
        self.arrivals.append(tag)
        if len(self.arrivals) == self.count:
            self.done, self.arrivals = self.arrivals, []
            self.phase += 1

    def passed(self, parity):
        return (self.phase & 1) != parity


def play(stages, new_words, period, tiles, rng, slow):
    """Plays tiles of the given k-block ranges; False where a round of a stage is counted full with arrivals of another round."""
    blocks, first = [], []
    for kb0, kb1 in tiles:
        for kb in range(kb0, kb1):
            blocks.append(kb)
            first.append(kb == kb0)
    total = len(blocks)
    full, empty = [Barrier(3) for _ in range(stages)], [Barrier(1) for _ in range(stages)]
    scale = [first[n] or blocks[n] % period == 0 for n in range(total)]      # the k-blocks that the scale warp takes part in
    assert all(scale[n] for n in range(total) if blocks[n] % new_words == 0)
    visits = [n for n in range(total) if scale[n]]
    at = {"weights": 0, "rows": 0, "scale": 0, "umma": 0, "release": 0}

    def ready(role):
        i = at[role]
        if role == "scale":
            if i == len(visits):
                return False
            n = visits[i]
            return empty[n % stages].passed((n // stages & 1) ^ 1)
        if i == total:
            return False
        if role == "umma":
            return full[i % stages].passed(i // stages & 1)
        if role == "release":
            return i < at["umma"]
        return empty[i % stages].passed((i // stages & 1) ^ 1)

    def act(role):
        i = at[role]
        at[role] += 1
        if role == "scale":
            full[visits[i] % stages].arrive(visits[i])
        elif role == "umma":
            return full[i % stages].done == [i] * 3
        elif role == "release":
            empty[i % stages].arrive(i)
        else:
            full[i % stages].arrive(i)
            if role == "weights" and not scale[i]:
                full[i % stages].arrive(i)
        return True

    while at["release"] < total:
        roles = [r for r in at if ready(r)]
        if not roles:
            return False                                   # everyone waits for everyone
        eager = [r for r in roles if r not in slow]
        if not act(rng.choice(eager if eager and rng.random() < 0.95 else roles)):
            return False
    return all(not b.arrivals and b.phase == len(range(s, total, stages)) for s, b in enumerate(full))


TILES = [[(0, 56)], [(0, 13), (0, 13), (0, 13)], [(3, 10), (10, 17), (0, 5)], [(0, 1)] * 9 + [(0, 6)]]
SLOW = [(), ("umma",), ("release",), ("scale",), ("weights",), ("rows",), ("umma", "scale"), ("release", "weights")]


@pytest.mark.parametrize("new_words", [1, 2, 4])
def test_every_round_of_a_stage_counts_its_own_arrivals(scale_period, new_words):
    for stages in range(1, most_stages() + 1):
        for tiles in TILES:
            for slow in SLOW:
                for seed in range(6):
                    assert play(stages, new_words, scale_period(stages, new_words), tiles, random.Random(seed), slow), (stages, tiles, slow, seed)


def test_long_rings_fetch_every_word_once(scale_period):
    # the rule's own tiles: the weight producer stands in for the scale warp on the k-blocks between, which saves that warp their re-ordering
    assert all(scale_period(s, p) == p for p in (1, 2, 4) for s in range(p, most_stages() + 1))


@pytest.mark.parametrize("stages,period", [(3, 4), (2, 4), (1, 4), (1, 2)])
def test_the_play_finds_rounds_mixed_up_where_visits_are_too_far_apart(stages, period):
    assert not all(play(stages, period, period, tiles, random.Random(seed), slow) for tiles in TILES for slow in SLOW for seed in range(6))
