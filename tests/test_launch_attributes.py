"""What the kernel launches ask of the CUDA runtime, on a stand-in with two
devices (tests/ffi/launch_probe.cpp): no GPU is needed."""

import os
import subprocess

import pytest

import build as native
from conftest import ROOT

OBJECTS = ("k_preprocess.cu.o", "k_tiles.cu.o", "k_sort.cu.o", "k_raster.cu.o")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    native.build()
    exe = str(tmp_path_factory.mktemp("probe") / "launch_probe")
    subprocess.run([native.CXX, "-std=c++17", "-O1", "-I", native.CSRC, "-I", native.INCLUDE,
                    "-I", os.path.join(native.CUDA_HOME, "include"),
                    os.path.join(ROOT, "tests", "ffi", "launch_probe.cpp"),
                    *[os.path.join(native.BUILD, o) for o in OBJECTS], "-o", exe], check=True)

    def lines(what, kind):
        out = subprocess.run([exe, what], capture_output=True, text=True, check=True).stdout
        return [line.split()[1:] for line in out.splitlines() if line.startswith(kind + " ")]

    def run(what):
        return [(int(d), int(smem), int(limit), prio)
                for d, smem, limit, prio in lines(what, "launch")]

    run.values = lambda what: [tuple(map(int, row)) for row in lines(what, what)]
    return run


@pytest.mark.parametrize("what", ["preprocess", "emit"])
def test_shared_memory_limits_are_raised_on_every_device(probe, what):
    """A kernel's dynamic shared memory limit belongs to a device: each device
    a process renders on has to get it, not the first one alone."""
    launches = probe(what)
    by_device = [[l[1:] for l in launches if l[0] == d] for d in (0, 1)]
    assert by_device[0] and by_device[0] == by_device[1]
    assert all(smem <= limit for _, smem, limit, _ in launches), launches


def test_sorts_keep_the_priority_of_their_stream(probe):
    """A sort asks for no priority unless its caller did: on a stream with a
    priority of its own every kernel of it then runs at that priority."""
    launches = probe("sort")
    assert len(launches) >= 2 * 9 and all(prio == "-" for *_, prio in launches), launches
    asked = probe("sort-high")
    assert asked and all(prio == "-5" for *_, prio in asked), asked


def test_admitted_pair_bytes_cover_the_workspace(probe):
    """What the server counts per pair is at least what a lane allocates: keys
    and values twice and the sort's scratch."""
    for capacity, words, counted in probe.values("work"):
        assert 16 * capacity + 4 * words <= counted * capacity + (1 << 16), (capacity, words)


def test_raster_shapes_are_what_is_launched(probe):
    """The autotuner compares candidates by the shape raster_shape names: equal
    shapes are one kernel on one grid, different ones are not. A chunk below
    the full tile is the step; the full tile's follows the number of tiles."""
    rows = set(probe.values("raster"))
    by_tiles = {}
    for tiles, mode, tile, chunk, bps, *shape, kernel, grid in rows:
        by_tiles.setdefault(tiles, set()).add((tuple(shape), kernel, grid))
        full = {16: 256 if tiles <= 7 * 148 else 128, 8: 128 if tiles <= 16 * 148 else 64}[tile]
        if mode == 0:
            assert shape[0] == (chunk if chunk < tile * tile else full)
        assert shape[2] == (0 if mode else bps)
    for pairs in by_tiles.values():
        assert len({s for s, *_ in pairs}) == len({k[1:] for k in pairs}) == len(pairs)


def test_raster_chunk_over_changes_of_the_tile_size(probe):
    """A chunk that was never set is the full tile at either tile size; one that
    was set stays where it is valid and becomes the full tile where it is not."""
    rows = {(tile, chunk): rest for tile, chunk, *rest in probe.values("raster-tile")}
    assert rows == {
        (16, 0): [64, 256, 0, 0], (16, 64): [64, 64, 3, 3], (16, 128): [64, 256, 3, 3],
        (16, 256): [64, 256, 3, 3], (8, 0): [256, 64, 0, 0], (8, 32): [256, 64, 3, 3],
        (8, 64): [64, 64, 3, 3]}
