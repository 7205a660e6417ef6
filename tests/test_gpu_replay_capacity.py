"""A history with more rows than the first pass has room for is replayed with
room, with every argument of the call: rows, counts and tallies are those of a
call that had the room at once."""

import numpy as np
import pytest

from conftest import golden
from test_elsepa import GROUP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elsepa", [False, True])
@pytest.mark.parametrize("sbethe", [False, True])
def test_replay_keeps_the_tables(elsepa, sbethe, cuda_device):
    from pyrite_b200 import simulate_trajectories
    from pyrite_b200.tables import ElsepaGroup, StoppingTables
    from test_gpu_transport import layers_of

    kw = dict(E0_keV=30.0, Ne=200, layers=layers_of(golden("transport_si30kev")), E_cut_keV=5.0, seed=4, lut=False,
              device=cuda_device, tallies=(16, 16))
    if elsepa:
        d = golden("elsepa_si30kev")
        kw.update(elastic_model="elsepa", elastic_tables=ElsepaGroup(*(d[f"el_{k}"] for k in GROUP)))
    if sbethe:
        d = golden("sbethe_si30kev")
        kw.update(stopping_tables=StoppingTables(d["sb_count"], d["sb_logE"], d["sb_logS"]))
    ref = simulate_trajectories(cap=4096, **kw)
    assert 8 < ref["seg_count"].max() <= 4096
    got = simulate_trajectories(cap=8, **kw)
    for k in ("seg_count", "exit_code", "final_E_keV", "r_mid", "v_hat", "L_ang", "E_keV", "elec_id", "tally_fates",
              "tally_exit_E", "tally_exit_theta"):
        assert np.array_equal(ref[k], got[k]), k
