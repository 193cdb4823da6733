"""The event-driven GR pass under load gives the same network, bit for bit, as the
plain GR pass: steps in which every MF spikes (more list items than an event CTA
lists at a time) and more than half of the GR do (more cells than a streaming CTA
lists at a time in some tile), more spike words than an event CTA has threads, every
size of event blocks, and more than 15 MF or GO inputs a cell, which are counted in
bytes, in one zone and in two and beside a network with few in a batch."""
import numpy as np
import pytest

import cbmtest

pytestmark = pytest.mark.gpu

# build_random_network's (gr_xp2, gr_yp2, go_xp2, go_yp2, mf_p2), its options
NETS = {
    "burst": ((9, 8, 5, 5, 11), dict(go_out_per_gr=4, mf_per_go=16, vel=147)),
    "burst_small": ((7, 7, 4, 4, 11), dict(go_out_per_gr=6, mf_per_go=8, vel=60)),
    "many_sources": ((9, 8, 5, 4, 13), dict(go_out_per_gr=4, mf_per_go=16, vel=60)),
    "half_million": ((10, 9, 5, 5, 10), dict(go_out_per_gr=4, mf_per_go=16, vel=147)),
    "wide": ((9, 8, 4, 4, 9), dict(go_out_per_gr=5, mf_per_go=8, vel=60, mf_per_gr=20, go_per_gr=17)),
    "wide_zones": ((10, 8, 4, 4, 9), dict(go_out_per_gr=3, mf_per_go=8, vel=40, mf_per_gr=16, go_per_gr=3, n_zones=2)),
}


def build(name):
    import cerebellum_simulation_b200 as cbm
    from cerebellum_simulation_b200 import networks
    dims, opt = NETS[name]

    def new_state(con, *args, **kw):  # room for 20 inputs a cell
        con = con.replace("maxnumpGRfromGOtoGR 4", "maxnumpGRfromGOtoGR 20")
        return cbm.CBMState.new(con.replace("maxnumpGRfromMFtoGR 4", "maxnumpGRfromMFtoGR 20"), *args, **kw)

    st = networks.build_random_network(*dims, networks.act_params("dense"), seed=11, new_state=new_state, **opt)
    if name.startswith("burst"):
        # MF input alone fires a GR: most of them spike when every MF does
        st.setActParam("gMFIncGR", 20 * st.act("gMFIncGR"))
        st.setActParam("gGOIncGR", 0.2 * st.act("gGOIncGR"))
    return st


def stream(name, steps):
    """10-60 Hz, with steps in which every MF spikes."""
    from cerebellum_simulation_b200 import networks
    mf = networks.uniform_mf_stream(1 << NETS[name][0][4], steps, seed=3, lo=10.0, hi=60.0)
    mf[[20, 21, 22, 23, 50]] = 1
    return mf


@pytest.mark.parametrize("name", sorted(NETS))
def test_event_pass_under_load(name, tmp_path, monkeypatch):
    import cerebellum_simulation_b200 as cbm
    path = str(tmp_path / "net.state")
    build(name).writeState(path)
    zones = NETS[name][1].get("n_zones", 1)
    mf = stream(name, 60)
    events = {1: [("plast", z, -0.002, 0.002) for z in range(zones)], 40: [("errdrive", 0, 1.0)]}

    def run(env):
        with monkeypatch.context() as m:
            for k, v in env.items():
                m.setenv(k, v)
            sim = cbm.CBMSimCore(cbm.CBMState(path), [3 + z for z in range(zones)], device=0)
        out, net, most = [], sim.getInputNet(), 0.0
        for a, b in ((0, 19), (19, 21), (21, 22), (22, 23), (23, 24), (24, 25), (25, 49), (49, 60)):
            cbmtest.product_run(sim, mf[a:b], events, t0=a, record=False)
            ap = net.exportAPGR()
            most = max(most, float(ap.mean()))
            out += [ap, net.exportGESumGR(), net.exportGISumGR(), net.exportVmGR(), net.exportSumGRInputGO()]
        sim.writeToState(str(tmp_path / "out.state"))
        out.append(np.fromfile(tmp_path / "out.state", dtype=np.uint8))
        kind = sim.pass_geometry()[0]
        sim.close()
        return kind, most, [np.array(x).copy() for x in out]

    kind, most, got = run({})
    assert kind == "grPassTmaKernel"
    if name.startswith("burst"):
        assert mf.shape[1] > 1024 and most > 0.5
    _, _, want = run({"CBM_PASS_TMA": "0"})
    for i, (x, y) in enumerate(zip(got, want)):
        assert x.tobytes() == y.tobytes(), (name, i)


def test_wide_network_in_a_batch(tmp_path, monkeypatch):
    import cerebellum_simulation_b200 as cbm
    paths = []
    for name in ("wide", "burst"):
        paths.append(str(tmp_path / f"{name}.state"))
        build(name).writeState(paths[-1])

    def run(env):
        with monkeypatch.context() as m:
            for k, v in env.items():
                m.setenv(k, v)
            states = [cbm.CBMState(p) for p in paths]
            b = cbm.CBMBatch(states, [[4 + i] for i in range(len(states))], device=0)
        for i, st in enumerate(states):
            b.set_eyelid_protocol(i, cbmtest.protocol_rates(st.con("numMF"), seed=i),
                                  **cbmtest.short_protocol(mfSeed=5 + i, numDataTrials=1))
        b.run(300, 20)
        out = []
        for i in range(len(paths)):
            b.writeToState(i, str(tmp_path / "out.state"))
            out.append(open(tmp_path / "out.state", "rb").read())
        return b.pass_geometry()[0], out

    kind, got = run({})
    assert kind == "grPassTmaKernel"
    assert got == run({"CBM_PASS_TMA": "0"})[1]
