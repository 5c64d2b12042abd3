"""Coupled rotors of unlike shapes against the oracle's system, FP64 bit for
bit: near wakes of different length (a sheet gathered for another rotor's sums
with that rotor's row count), three lifting rotors, and bound-vortex sums over
more panels than a batch holds and more blades than a group takes."""
import pytest

from test_gpu_system import assert_same_state, gpu_system, oracle_system
from volcanor_gb300 import cases as C

pytestmark = pytest.mark.gpu


def run(geoms, steps):
    pair = C.rotor_pair(nt=steps)
    sc = C.SystemCase("rotors", pair.config.replace("nr = 2", f"nr = {len(geoms)}"), geoms)
    o = oracle_system(sc, steps)
    g, _ = gpu_system(sc, steps)
    for ir in range(len(geoms)):
        assert_same_state(g.rotors[ir], o.rotors[ir], o.rotors[ir].geti("nb"))


def rotor(z, omega, rows, truncate, **shape):
    return C.rotor_pair(nt=2, n_nwake=rows, truncate_nt=truncate, hub2=(0.0, 0.0, z), omega2=omega, **shape).geoms[1]


@pytest.mark.parametrize("rows", [(5, 9), (9, 5), (4, 7, 6)])
def test_unequal_near_wakes(rows):
    run([rotor(-0.3 * i, 100.0 if i % 2 == 0 else -100.0, r, r + 3, ns=5 + i) for i, r in enumerate(rows)], 14)


def test_many_panels_and_many_blades():
    run([rotor(0.0, 100.0, 3, 0, nc=16, ns=17), rotor(-0.3, -100.0, 3, 0, nb=34, ns=2)], 3)
