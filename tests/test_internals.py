"""Decisions of the library's host code: memory admission, the autotuner's candidates and
what a serving slot is given ahead of its first batch."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def internals(tmp_path_factory):
    from saq_gb300.build import LIB, NVCC, build
    build()
    exe = str(tmp_path_factory.mktemp("internals") / "internals")
    cuda = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, os.path.join(ROOT, "tests", "internals.cpp"),
                    "-I", os.path.join(ROOT, "saq_gb300", "csrc"), "-isystem", cuda, LIB,
                    f"-Wl,-rpath,{os.path.dirname(LIB)}", "-lpthread"], check=True)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True)
        return [[int(v) for v in line.split()] for line in r.stdout.splitlines()]
    return run


@pytest.mark.parametrize("segs", [1, 2, 4, 16])
def test_admission_counts_two_thirds_of_the_records(internals, segs):
    """A batch is admitted with the record space that a record without its 32 ids took (the
    ids came later: 128 bytes), 8 GB at most; a few queries with all of it."""
    record = 4 * (8 + segs + 1 + 32 + 32 * segs) + 16  # header, stage minima, estimates, partials; summary
    k, np, step = 10, 32, 20

    def slope(nq):  # bytes counted per block of a query
        a, b = (internals("estimate", segs, blocks, nq, k, np)[0][0] for blocks in (step, 2 * step))
        return (b - a) / (nq * np * step)
    assert slope(256) <= record + 16  # up to rounding to whole words
    assert record + 128 <= slope(8) <= record + 160
    most = [internals("estimate", segs, blocks, 4096, k, np)[0][0] for blocks in (2000, 20000)]
    assert most[0] == most[1]  # bounded
    none = internals("estimate", segs, 1, 4096, k, np)[0][0]
    assert most[0] - none <= 8 << 30


def test_autotuner_tries_every_level_set_at_the_built_in_line(internals):
    cands = internals("candidates")
    assert cands[0] == [-1, -1, -1, -1]
    for levels in (1, 2, 3, 4):
        assert any(mode == 0 and defer == -1 and lv == levels for mode, defer, _, lv in cands)


@pytest.mark.gpu
def test_tensor_core_slot_has_its_streams(internals, golden_case_by_name):
    """A context sized ahead for the tensor-core form has the streams and events that form
    forks onto, so its first batch creates none."""
    from conftest import INDEX_CASES
    assert internals("presize", golden_case_by_name(INDEX_CASES[0])) == [[1] * 6]


def test_only_a_few_queries_get_short_tiles(internals):
    for mode, nq, blocks in internals("tiles"):
        assert blocks == (4 if mode == 1 and nq <= 16 else 16)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 60000, 125000, 1000003])
def test_encoder_chunks_fit_one_wave_at_every_width(internals, n):
    held = []
    for bits, chunk, at_once in internals("chunks", n, 512):
        assert chunk % 32 == 0 and 32 <= chunk <= at_once
        assert chunk >= min(n, at_once) / 2 - 32  # equal shares, not a full one and a rest
        held.append(at_once)
    assert min(held) < max(held)  # 6-bit codes keep their values in a larger table
