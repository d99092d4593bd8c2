"""The tuning table of tile sizes: its lines set the slots of the classes they name; a table from before
there were tiles, whose lines of three numbers count a chunk's entries, sets none."""
import pytest

from conftest import flat_of, squeezed_lattice

pytestmark = pytest.mark.gpu


def cap(flat, precision):
    from melody2d_b200.solver import Solver
    s = Solver.from_flat(flat, precision=precision)
    c = s.kernel_config()["chunk_cap"]
    s.close()
    return c


@pytest.mark.parametrize("table,fp64,mixed", [
    ("# chunks\n0 404 2048\n1 404 3328\n0 576 1792\n1 576 2816\n", None, None),
    ("# tiles\ntile 0 404 2048\ntile 1 404 4608\n", 2048, 4608),
    ("tile 0 100 2048\n0 404 2304\ntile 0 404 2560\ntile 1 404 99999\n", 2560, None)])
def test_table_lines(gpu_lib, monkeypatch, tmp_path, table, fp64, mixed):
    flat = flat_of(squeezed_lattice(2, 2))
    path = tmp_path / "table.txt"
    path.write_text("")
    monkeypatch.setenv("MELGPU_TUNE_FILE", str(path))
    rule = [cap(flat, 0), cap(flat, 1)]
    assert rule[0] > 2560
    path.write_text(table)
    assert cap(flat, 0) == (fp64 or rule[0])
    assert cap(flat, 1) == (mixed or rule[1])
