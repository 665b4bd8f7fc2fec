"""Which tile height a single grid's launches use (kernels.cu tile_rows): fewer rows
where the tiles then still fit the same rounds of the SMs, full tiles where only
17 or 18 of the 19 rows would (that costs time instead of saving it)."""
import pytest

pytestmark = pytest.mark.gpu

# One size of each kind, for 148 SMs.
ROWS = [(64, 2), (128, 4), (192, 8), (256, 15), (320, 12), (352, 14), (384, 16), (448, 15), (480, 19),
        (288, 19), (576, 19), (640, 19), (768, 19), (512, 19)]


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_tile_rows_by_grid_size(pmhd_lib, precision):
    torch = pytest.importorskip("torch")
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are chosen for 148 SMs")
    got = []
    for n, _ in ROWS:
        with pmhd_lib.Solver(nx=n, ny=n, precision=precision) as s:
            s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
            got.append((n, s.advance(max_steps=2).tile_height))
    assert got == ROWS
