"""The event-driven GR pass (the default one) gives the same network, bit for
bit, as the plain GR pass at the edges of its tables: tiles of part of a row, of
whole rows and of several PCs; one event block and several; no spare slot (15 MF
and 15 GO inputs a cell, the most a count holds) and one more (which runs the
plain pass); more GR->GO synapses than a table row; delays of 0, which are
delivered in their own step, and up to 31; two microzones; few and many sources.
The plain kernel is pinned to the oracle by test_gpu_parity.py."""
import numpy as np
import pytest

import cbmtest

pytestmark = pytest.mark.gpu

# build_random_network's (gr_xp2, gr_yp2, go_xp2, go_yp2, mf_p2), its options
NETS = {
    "small": ((7, 5, 2, 2, 5), dict(go_out_per_gr=1, mf_per_go=4, vel=40, sc_p2=5)),
    "one_block": ((8, 6, 4, 4, 10), dict(gr_per_go=128, mf_per_go=3, vel=40)),
    "full_counts": ((7, 6, 4, 4, 9), dict(go_out_per_gr=3, mf_per_go=4, vel=20, mf_per_gr=15, go_per_gr=15)),
    "over_counts": ((7, 6, 4, 4, 9), dict(go_out_per_gr=3, mf_per_go=4, vel=20, mf_per_gr=16, go_per_gr=3)),
    "many_outputs": ((9, 7, 4, 4, 7), dict(go_out_per_gr=13, mf_per_go=8, vel=9)),
    "delay_zero": ((9, 7, 3, 3, 7), dict(go_out_per_gr=5, mf_per_go=8, vel=60, af_delay=0)),
    "two_zones": ((9, 8, 5, 5, 11), dict(go_out_per_gr=4, mf_per_go=16, vel=147, n_zones=2)),
    "many_pcs": ((9, 8, 5, 4, 9), dict(go_out_per_gr=4, mf_per_go=8, vel=30, pc_p2=7)),
}


@pytest.mark.parametrize("name", sorted(NETS))
def test_event_pass_matches_plain_pass(name, tmp_path, monkeypatch):
    import cerebellum_simulation_b200 as cbm
    from cerebellum_simulation_b200 import networks
    dims, opt = NETS[name]

    def new_state(con, *args, **kw):  # room for 16 inputs a cell
        con = con.replace("maxnumpGRfromGOtoGR 4", "maxnumpGRfromGOtoGR 16")
        return cbm.CBMState.new(con.replace("maxnumpGRfromMFtoGR 4", "maxnumpGRfromMFtoGR 16"), *args, **kw)

    st = networks.build_random_network(*dims, networks.act_params("dense"), seed=11, new_state=new_state, **opt)
    path = str(tmp_path / "net.state")
    st.writeState(path)
    zones = opt.get("n_zones", 1)
    mf = networks.uniform_mf_stream(1 << dims[4], 110, seed=3, lo=10.0, hi=90.0)
    events = {1: [("plast", z, -0.002, 0.002) for z in range(zones)], 40: [("errdrive", 0, 1.0)]}

    def run(env):
        with monkeypatch.context() as m:
            for k, v in env.items():
                m.setenv(k, v)
            sim = cbm.CBMSimCore(cbm.CBMState(path), [3 + z for z in range(zones)], device=0)
        out, net = [], sim.getInputNet()
        # exports between steps read the arrays while the pass runs them
        for a, b in ((0, 1), (1, 37), (37, 110)):
            cbmtest.product_run(sim, mf[a:b], events, t0=a, record=False)
            out += [net.exportGESumGR(), net.exportGISumGR(), net.exportVmGR(), net.exportAPBufGR(),
                    net.exportSumGRInputGO(), net.exportHistoryGR()]
            out += [z.exportPFPCWeights() for z in sim.getMZoneList()]
            sim.writeToState(str(tmp_path / "out.state"))
            out.append(np.fromfile(tmp_path / "out.state", dtype=np.uint8))
        kind = sim.pass_geometry()[0]
        sim.close()
        return kind, [np.array(x).copy() for x in out]

    kind, got = run({})
    assert kind == ("grPassKernel" if name == "over_counts" else "grPassTmaKernel")
    _, want = run({"CBM_PASS_TMA": "0"})
    assert want[-zones - 4].any()  # GR cells spike (APBuf of the last part)
    for i, (x, y) in enumerate(zip(got, want)):
        assert x.tobytes() == y.tobytes(), (name, i)
