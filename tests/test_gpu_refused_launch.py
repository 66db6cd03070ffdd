"""A kernel launch that the runtime refuses while a substep is captured: pbf_step reports
it, no graph without that kernel runs, and the next call captures anew. (The refused
launch is one of an empty grid, which fails on the host.)"""
import pytest

from oracle import oracle as O
from pbf_b200 import Solver, scenes
from pbf_b200._lib import PBF_ERR_CUDA, PBF_ERR_INVALID, PBFError, check, lib

from helpers import mismatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adaptive", [0, 1])
@pytest.mark.parametrize("block,persistent", [(12, 0), (12, 1)])
def test_refused_launch_is_reported(block, persistent, adaptive):
    sc = scenes.dam_break(block, (40, 20, 20), stable=True, iterations=2)
    s = Solver(sc.para, sc.grid_space, sc.boundary,
               sc.ext(adaptive=adaptive, density_tol=1e-9, max_iterations=2, persistent=persistent))
    s.upload(sc.pos, sc.vel)
    # scatter, reorder, search, two lambda and two delta-p passes, curl, vorticity
    for k in range(1, 10):
        check(lib().pbf_debug_fail_launch(k))
        try:
            with pytest.raises(PBFError) as e:
                s.step(1)
        finally:
            check(lib().pbf_debug_fail_launch(0))
        assert e.value.code == PBF_ERR_CUDA and "launches" in str(e.value), (k, str(e.value))
    s.step(2)
    assert s.stats()["error_bits"] == 0
    orc = O.Oracle(O.params_for_scene(sc), sc.pos, sc.vel)
    orc.substep(2)
    for f in ("x", "v"):
        assert mismatch(s.fetch(f)[:, :3], orc.get(f))[0] == 0, f
    s.close()
    orc.close()
    assert lib().pbf_debug_fail_launch(-1) == PBF_ERR_INVALID
