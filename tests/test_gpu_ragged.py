"""The dense passes and the compaction at sizes around their words, chunks and
warps, the pool at and beyond the grid's faces, against the CPU oracle."""
import pytest

from test_gpu_parity import run_and_compare

pytestmark = pytest.mark.gpu

DECK = """dx 4.0e-6
nX %d %d %d
bmV 1.0
bmP 180.0
bmDelT 25e-6
r 4e-3
lT 20e-6
bpH 28e-6
tL 1609
tS 1531.5
meltparam 30e-6 90e-6 30e-6 28e-6
bhatch 3.0e-5
mu .006
lrate .0009
patternID 2
outint 1
offset %g -10.0e-6 0.0
gridsize 1.6e-4 1.2e-4
gridtheta %g
dendritegrowth2 0.0001 2.0
"""


@pytest.mark.parametrize("theta", [0.0, 0.7])
@pytest.mark.parametrize("nx,ny,nz", [(5, 7, 12), (8, 5, 12), (9, 16, 13), (31, 3, 12), (32, 4, 14), (33, 9, 12),
                                      (64, 5, 12), (65, 6, 13), (130, 8, 12)])
def test_ragged_grids(tmp_path, nx, ny, nz, theta):
    path = tmp_path / "ragged.in"
    path.write_text(DECK % (nx, ny, nz, -20e-6, theta))
    run_and_compare(str(path), 0, 3, tmp_path)


@pytest.mark.parametrize("mu,lrate", [("1e-6", "1e-6"), ("2e-4", ".0009"), (".2", ".1")])
@pytest.mark.parametrize("nx,ny,nz", [(33, 9, 12), (130, 8, 12), (20, 21, 40)])
def test_grain_densities(tmp_path, nx, ny, nz, mu, lrate):
    """from one grain for the whole baseplate to more grains than cells"""
    path = tmp_path / "ragged.in"
    text = DECK % (nx, ny, nz, -20e-6, 0.7)
    path.write_text(text.replace("mu .006", "mu " + mu).replace("lrate .0009", "lrate " + lrate))
    run_and_compare(str(path), 0, 5, tmp_path)
