"""The library's work is ordered by its own streams: with another library's
kernels queued on the default stream the whole time, a simulator built, switched to
its recording protocol, stepped, recorded and exported gives the bytes that it gives
on an idle device."""
import contextlib
import threading

import numpy as np
import pytest

import cbmtest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def busy_default_stream():
    """Kernels of about 2 ms queued behind one another on the default stream."""
    import torch
    stop = threading.Event()
    torch.cuda.synchronize()
    torch.cuda._sleep(1000)

    def feed():
        while not stop.is_set():
            ends = []
            for _ in range(4):  # at most 8 ms are queued
                torch.cuda._sleep(3000000)
                ends.append(torch.cuda.Event())
                ends[-1].record()
            ends[1].synchronize()

    t = threading.Thread(target=feed)
    t.start()
    try:
        yield
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize()


def test_simulator_beside_default_stream_work(tmp_path):
    import cerebellum_simulation_b200 as cbm
    from cerebellum_simulation_b200 import networks
    # several GR->GO synapses a cell: rows of the overflow table are in use
    st = networks.build_random_network(9, 8, 5, 5, 10, networks.act_params("dense"), seed=5,
                                       go_out_per_gr=9, mf_per_go=16, vel=60)
    path = str(tmp_path / "net.state")
    st.writeState(path)
    mf = networks.uniform_mf_stream(1024, 60, seed=5, lo=10.0, hi=90.0)
    rates = cbmtest.protocol_rates(1024, seed=4)
    proto = cbmtest.short_protocol(mfSeed=9)

    def run():
        sim = cbm.CBMSimCore(cbm.CBMState(path), [3], device=0)
        cbmtest.product_run(sim, mf, {1: [("plast", 0, -0.002, 0.002)]}, record=False)
        net, zone = sim.getInputNet(), sim.getMZoneList()[0]
        out = [net.exportAPGR(), net.exportGESumGR(), net.exportVmGR(), zone.exportPFPCWeights()]
        sim.set_eyelid_protocol(rates, **proto)
        sim.record_gr()
        sim.record_trial_data()
        sim.run(2 * proto["trialSteps"], 20)
        out += [sim.trial_record(k) for k in ("nc", "pc", "gr")]
        sim.writeToState(str(tmp_path / "out.state"))
        out.append(np.fromfile(tmp_path / "out.state", dtype=np.uint8))
        sim.close()
        return [np.array(x).tobytes() for x in out]

    want = run()
    for k in range(3):
        with busy_default_stream():
            got = run()
        assert [a == b for a, b in zip(got, want)] == [True] * len(want), k


def test_surrogate_beside_default_stream_work():
    """Parameters set, then trained on at once: Adam starts from zero moments."""
    from cerebellum_simulation_b200.surrogate import MLP
    rng = np.random.Generator(np.random.PCG64(8))
    x = rng.uniform(-1, 1, (512, 24)).astype(np.float32)
    t = rng.uniform(0, 2, (512, 10)).astype(np.float32)

    def run(busy):
        net = MLP(24, 96, 64, 10, max_batch=128, seed=2)
        start = net.get_params()
        net.train(x, t, batch=128, epochs=2, lr=1e-2, seed=1)  # leaves moments behind
        with busy_default_stream() if busy else contextlib.nullcontext():
            net.set_params(start)
            net.train(x, t, batch=128, epochs=2, lr=1e-2, seed=1)
            return net.get_params().tobytes()

    want = run(False)
    for _ in range(3):
        assert run(True) == want
