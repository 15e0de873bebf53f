"""A checkpoint holds the scene's state and nothing of what its read-outs left behind."""
import pytest

import campfire_b200 as cb
from campfire_b200.fluid import load_scene

pytestmark = pytest.mark.gpu


def test_reads_leave_the_checkpoint_as_it_is(tmp_path):
    # U of 224x320 cells is padded and larger than the staging area: it is packed in the scene's spare array
    nx, ny = 224, 320
    sc = cb.generate_scene(0, nx, ny, 0.8, 5)
    g = cb.FluidSim(0, {"nx": nx, "ny": ny, "dt": sc["dt"]}, width=0.8).init()
    load_scene(g, sc)
    g.step(1)
    g.save_checkpoint(str(tmp_path / "a"))
    for f in ("U", "T", "Y", "fx"):
        g.readBuffer(f)
    g.save_checkpoint(str(tmp_path / "b"))
    assert (tmp_path / "a").read_bytes() == (tmp_path / "b").read_bytes()
    # radiation's result is state, its emission per cell is not
    rad = g.readBuffer("rad")
    g.encodeRadiation()
    g.writeBuffer("rad", rad)
    g.save_checkpoint(str(tmp_path / "c"))
    g.close()
    assert (tmp_path / "a").read_bytes() == (tmp_path / "c").read_bytes()
