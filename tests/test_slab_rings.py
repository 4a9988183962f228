"""The depths of the slab-fed GEMM's rings (csrc/slab_rings.h, host code) over every slab size, weight stage and stage count."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fastertnn_b200" / "csrc"
AVAIL = 232448 - 1024 - 512  # shared memory of a block less alignment and barriers
COPIES, LOADERS, LOADERS_TWO = 0, 1, 2
MAXSLAB, MAXSTG = 8, 12
SLABS = range(1024, 65536 + 1, 1024)


@pytest.fixture(scope="module")
def rings(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("rings")
    (d / "r.cpp").write_text('#include "slab_rings.h"\nextern "C" int rings(int slab, int stage, int avail, int n, int one, int feed, int* out) {\n'
                             "    SlabRings r;\n    if (!slab_rings(slab, stage, avail, n, one != 0, (SlabFeed)feed, &r)) return 0;\n"
                             "    out[0] = r.nslab; out[1] = r.nstg; out[2] = r.resident;\n    return 1;\n}\n")
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "r.cpp"), "-o", str(d / "r.so")], check=True)
    fn = C.CDLL(str(d / "r.so")).rings

    def call(slab, stage, nchunks, one_kernel_tile, feed):
        out = (C.c_int * 3)()
        return tuple(out) if fn(slab, stage, AVAIL, nchunks, int(one_kernel_tile), feed, out) else None
    return call


@pytest.mark.parametrize("feed", [COPIES, LOADERS, LOADERS_TWO])
def test_rings_fit(feed, rings):
    for slab in SLABS:
        for stage in (8192, 16384, 32768):
            for nchunks in range(1, 20):
                for one in (False, True):
                    r = rings(slab, stage, nchunks, one, feed)
                    assert (r is None) == (2 * slab + 3 * stage > AVAIL), (slab, stage, nchunks, one)
                    if r is None:
                        continue
                    ns, nb, stays = r
                    assert 2 <= ns <= MAXSLAB and 1 <= nb <= MAXSTG and ns * slab + nb * stage <= AVAIL
                    assert nb == nchunks if stays else nb >= 3
                    assert not stays or one
                    # loaders and two issuers take the slabs in turn
                    assert feed == COPIES or ns % 2 == 0


def test_two_issuers_use_the_memory_there_is(rings):
    """As many slabs as leave the weights resident, whatever a slab's size."""
    for slab in SLABS:
        for nchunks in (3, 5):  # 64 and 128 channels
            ns, nb, stays = rings(slab, 8192, nchunks, True, LOADERS_TWO)
            assert stays and nb == nchunks
            assert ns == MAXSLAB or (ns + 2) * slab + nchunks * 8192 > AVAIL, slab


def test_loaders_displace_no_weights_that_could_stay(rings):
    """Weights that fit beside two slabs stay; four slabs of tensor copies are no reason to stream them either."""
    for feed in (LOADERS, LOADERS_TWO):
        for slab in SLABS:
            for stage in (8192, 16384, 32768):
                for nchunks in range(3, MAXSTG + 1):
                    r = rings(slab, stage, nchunks, True, feed)
                    if r:
                        assert r[2] == (2 * slab + nchunks * stage <= AVAIL), (feed, slab, stage, nchunks)


@pytest.mark.parametrize("stage", [8192, 16384, 32768])
def test_ring_of_weights_is_sized_for_the_slabs_that_are_kept(stage, rings):
    """Streamed weights get what the slabs leave: another stage would not fit."""
    for feed in (COPIES, LOADERS, LOADERS_TWO):
        for slab in SLABS:
            r = rings(slab, stage, 40, False, feed)
            if r:
                assert r[1] == MAXSTG or r[0] * slab + (r[1] + 1) * stage > AVAIL, (feed, slab)
