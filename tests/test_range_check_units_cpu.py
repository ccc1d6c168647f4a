"""Range-checked builds: the recorded violation is per translation unit, so every
unit that compiles kernels with checks has a reader that the query calls."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qimpy_gb300", "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_every_unit_with_checked_kernels_is_read():
    units = [os.path.basename(p)[:-3] for p in glob.glob(os.path.join(CSRC, "*.cu"))]
    checked = [u for u in units if re.search(r"^template int launch_", _text(u + ".cu"), re.M)]
    assert {"local_f32", "local_f64", "batched_f32", "batched_f64", "density_f32", "density_f64"} <= set(checked)
    query = re.search(r"int debug_violation\(.*?\n}", _text("local_potential.cu"), re.S).group(0)
    for u in checked:
        assert f"int violation_{u}(" in _text(u + ".cu"), u
        assert f"violation_{u}" in query, u


def test_points_are_checked_before_their_tables_are_read():
    """A sphere point's index is tested where it is first used, not after the loads."""
    body = _text("local_kernels.cuh")
    assert len(re.findall(r"g < g1 && QGB_OK_IDX\(g, s\.n\[k\], 1\)", body)) == 2
    for site in (4, 5, 6, 8):  # planes of the y/z passes and of the x-pass, its slabs, V
        assert re.search(rf"QGB_OK_IDX\([^;]*, {site}\)", body), site
