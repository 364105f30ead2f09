"""Guided inpainting against the CPU oracle.

Once the locked pixels outnumber the ones to synthesise the guide's weight is
negative (ms.rs:853-858), so a partial cost can fall again: the result must
still be the reference's sequential one, whatever launch shape resolves it.
"""
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [48, 64])
@pytest.mark.parametrize("team,full", [(None, 256), (0, 0), (1 << 30, 0)])
def test_guided_inpaint(ts, oracle, wl, side, team, full):
    spec = wl.inpaint_session(11, side=side)
    spec["examples"][0]["guide"] = wl.example_guide(5, side, side, sigma=2.0)
    spec["target_guide"] = wl.target_guide(6, side, side)
    got = ts.run_spec(spec, team_max_batch=team, team_full_max_batch=full)
    assert_same(got, oracle.run(spec, nthreads=4), "guided inpaint %d^2" % side)
