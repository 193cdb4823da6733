"""Networks with few and many NC and IO cells in one and several microzones: every
step matches the oracle, and the NC spikes read straight after a single step (from
the mailbox: in one word with the step number up to 16 of them, as bytes behind it
beyond) are those of the device's spike buffers."""
import numpy as np
import pytest

import cbmtest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc_p2,io_p2,zones", [(0, 0, 1), (3, 2, 1), (4, 2, 1), (3, 2, 2), (5, 3, 1), (3, 2, 4), (4, 4, 2)])
def test_steps_match_oracle(nc_p2, io_p2, zones, tmp_path):
    import cerebellum_simulation_b200 as cbm
    from cerebellum_simulation_b200 import networks
    st = networks.build_random_network(7, 7, 4, 4, 9, networks.act_params("dense"), seed=3, go_out_per_gr=4, mf_per_go=8,
                                       vel=60, nc_p2=nc_p2, io_p2=io_p2, n_zones=zones)
    path = str(tmp_path / "net.state")
    st.writeState(path)
    seeds = [21 + z for z in range(zones)]
    mf = networks.uniform_mf_stream(512, 130, seed=7, lo=20.0, hi=100.0)
    events = {1: [("plast", z, -0.002, 0.002) for z in range(zones)], 40: [("errdrive", zones - 1, 1.0)]}
    oracle = cbmtest.Oracle(path, seeds=seeds)
    want = oracle.run(mf, events)
    sim = cbm.CBMSimCore(cbm.CBMState(path), seeds, device=0)
    got, spikes = [], 0
    for t in range(len(mf)):
        cbmtest.product_run(sim, mf[t:t + 1], events, t0=t, record=False)
        nc = [z.exportAPNC().copy() for z in sim.getMZoneList()]  # before anything else is read
        for z, ap in zip(sim.getMZoneList(), nc):
            assert np.array_equal(ap, z.exportAPBufNC() & 1), t
            spikes += int(ap.sum())
        got.append(cbmtest.product_record(sim, None))
    assert spikes > 0
    assert cbmtest.first_difference(want, np.stack(got), oracle.num) is None
