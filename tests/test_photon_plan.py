"""How SPPM's photons are cut into waves (csrc/photon_plan.cuh, compiled here
with g++): passes over an iteration, and the memory a wave asks for."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ajisai_render_gb300" / "csrc"
QUEUE, RECORD = 112, 52  # bytes of a photon's queue entries, of a deposit record
LIMIT = 1 << 25          # records of a wave


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(
        '#include "photon_plan.cuh"\n'
        'extern "C" void plan(uint64_t n, uint64_t it, int depth, uint64_t most, int tries,\n'
        '                     uint64_t* o) {\n'
        '  const ajg::PhotonPlan p = ajg::photon_plan(n, it, depth, most, tries);\n'
        '  o[0] = p.chunk; o[1] = p.group; o[2] = p.depths; o[3] = p.records;\n'
        '}\n')
    out = d / "plan.so"
    r = subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC),
                        str(d / "plan.cpp"), "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(out))
    lib.plan.argtypes = [C.c_uint64, C.c_uint64, C.c_int, C.c_uint64, C.c_int, C.c_void_p]

    def f(n, it, depth, most, tries=0):
        o = (C.c_uint64 * 4)()
        lib.plan(n, it, depth, most, tries, o)
        return list(o)
    return f


CASES = [(n, it, depth, most)
         for n in (0, 1, 33, 100_000, 2_000_000, 50_000_000)
         for it in (1, 7, 100) for depth in (0, 1, 2, 10, 64, 128, 1024)
         for most in (1024, 1 << 20, 1 << 28)]


def test_an_iteration_takes_no_more_passes_than_its_photons_need(plan):
    for n, it, depth, most in CASES:
        chunk, group, depths, records = plan(n, it, depth, most)
        assert -(-n // chunk) == -(-n // most), (n, it, depth, most)
        assert records == chunk * depths and depths <= max(0, depth - 1)
        assert 1 <= group <= it
        # every photon of a wave may deposit at each of the depths
        assert records * group <= max(LIMIT, chunk)
        if depth > 1:
            assert depths >= 1
        if group > 1:  # held until the iterations' own grids stand
            assert depths == max(0, depth - 1) and -(-n // chunk) == 1


def test_failed_allocations_end_below_what_the_photons_alone_take(plan):
    """The queues of min(photons, wave) photons are what a render needs
    without any records: some try asks for no more."""
    for n, it, depth, most in CASES:
        alone = QUEUE * max(1, min(n, most))
        last = None
        for tries in range(64):
            chunk, group, depths, records = plan(n, it, depth, most, tries)
            assert group == 1 or tries == 0
            if depth > 1:
                assert depths >= 1 and records == chunk * depths
            need = QUEUE * chunk * group + RECORD * records * group
            assert last is None or need <= last
            last = need
            if tries and chunk == 1:
                break
        assert chunk == 1
        assert need <= max(alone, QUEUE + RECORD * max(0, depth - 1)), (n, it, depth, most)
