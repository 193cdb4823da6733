"""Performance cases: what a user of this framework has it do.

Simulations of the cerebellar network in the sizes of this repository's
configurations (16K, 256K to 2M, 1M and dense 4M granule cells), stepped one
call at a time as the reference's driver does, run in chunks from resident
input, run as whole recorded eyelid sessions, and batched; the surrogate MLP's
inference, gradients and training; and the allocation-free PF->PC sums.

A simulating case keeps one network (its wiring is part of the case, as a
user keeps one network over many runs); the seed gives its initial PF->PC
weights, its mossy-fibre input and its transmitter-release draws.
"""
import ctypes
import functools
import io

import numpy as np
import torch

import cerebellum_simulation_b200 as cbm
from cerebellum_simulation_b200 import networks, sweep
from cerebellum_simulation_b200.surrogate import MLP

# GR count (log2) -> GR grid exponents, and GO grid exponents, of the random
# networks with 4 GO targets per GR
GRIDS = {14: (8, 6), 15: (8, 7), 16: (9, 7), 17: (9, 8), 18: (10, 8), 19: (10, 9), 20: (11, 9), 21: (11, 10)}


def listed():
    return [
        # a closed-loop controller on the small network: one call per 1 ms
        # step, the nucleus read after each (the smallest calls)
        {"name": "loop_16k", "kind": "loop", "net": "c1", "steps": 16},
        # the same on the 1M eyelid network
        {"name": "loop_1m", "kind": "loop", "net": "c2", "steps": 64},
        # the 16K network over a stretch of resident input
        {"name": "run_16k", "kind": "run", "net": "c1", "steps": 500, "chunk": 50},
        # the 1M eyelid network, the headline configuration, with learning on
        {"name": "run_1m", "kind": "run", "net": "c2", "steps": 1000, "chunk": 50},
        # the dense 4M network under cart-pole-style state coding on the device
        {"name": "run_dense4m", "kind": "dense", "net": "c3", "steps": 200, "chunk": 50},
        # an eyelid session with every record the driver keeps
        {"name": "session_256k", "kind": "session", "p2": 18, "trial": 500, "trials": 2, "bin": 10, "chunk": 50},
        # a parameter sweep of the 16K network (the surrogate's training data)
        {"name": "sweep_16k_x64", "kind": "sweep", "n": 64, "steps": 500, "chunk": 250},
        # uneven instances in one launch (GR counts 2^p2), one eyelid protocol each
        {"name": "batch_uneven", "kind": "batch", "p2": "18,21,19,20,18,19", "steps": 100, "chunk": 50},
        # ranking sweep candidates with the surrogate
        {"name": "mlp_forward", "kind": "forward", "sizes": "64,256,256,50", "rows": 4096, "max_batch": 256},
        # one odd-sized minibatch's gradients
        {"name": "mlp_gradients", "kind": "gradients", "sizes": "64,256,256,50", "rows": 200, "max_batch": 256},
        # an epoch of training the surrogate
        {"name": "mlp_train", "kind": "train", "sizes": "64,256,256,50", "rows": 4096, "max_batch": 256, "batch": 256},
        # PF->PC sums on a caller's own buffers (1M fibres, 32 PCs)
        {"name": "pfpc_1m", "kind": "pfpc", "pcs": 32, "fibres": 32768},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["loop", "run", "session", "sweep", "batch", "forward", "gradients", "train", "pfpc"])
    if kind in ("loop", "run"):
        p2 = rng.randint(14, 20)
        if kind == "loop":
            return {"kind": kind, "net": str(p2), "steps": _log_int(rng, 8, 64)}
        return {"kind": kind, "net": str(p2), "steps": _log_int(rng, 100, 1000), "chunk": _log_int(rng, 10, 100)}
    if kind == "session":
        return {"kind": kind, "p2": rng.randint(14, 18), "trial": rng.randint(300, 700), "trials": rng.randint(1, 2),
                "bin": rng.randint(7, 25), "chunk": rng.randint(20, 100)}
    if kind == "sweep":
        return {"kind": kind, "n": _log_int(rng, 4, 64), "steps": _log_int(rng, 100, 500), "chunk": rng.randint(25, 250)}
    if kind == "batch":
        p2 = [rng.randint(17, 20) for _ in range(rng.randint(2, 4))]
        return {"kind": kind, "p2": ",".join(map(str, p2)), "steps": rng.randint(50, 100), "chunk": rng.randint(10, 50)}
    if kind == "pfpc":
        fibres = 1 << rng.randint(5, 15)
        return {"kind": kind, "pcs": rng.randint(3, 128), "fibres": fibres}
    sizes = "%d,%d,%d,%d" % (rng.randint(6, 64), rng.randint(32, 256), rng.randint(32, 256), rng.randint(5, 64))
    if kind == "forward":
        return {"kind": kind, "sizes": sizes, "rows": _log_int(rng, 1, 4096), "max_batch": rng.randint(64, 512)}
    mb = rng.randint(64, 512)
    if kind == "gradients":
        return {"kind": kind, "sizes": sizes, "rows": rng.randint(1, mb), "max_batch": mb}
    return {"kind": kind, "sizes": sizes, "rows": _log_int(rng, mb, 4096), "max_batch": mb, "batch": rng.randint(32, mb)}


# ------------------------------------------------------------------ networks
@functools.lru_cache(maxsize=None)
def _image(net):
    """State-file bytes of a configuration's network ("c1" 16K, "c2" 1M, "c3"
    dense 4M) or of the random network of 2^net GR."""
    if net == "c1":
        st = networks.config1_network(seed=0)
    elif net == "c2":
        st = networks.config2_network(seed=0)
    elif net == "c3":
        st = networks.config3_network(seed=0)
    else:
        gx, gy = GRIDS[int(net)]
        go = (4, 4) if int(net) < 17 else (6, 4)
        st = networks.build_random_network(gx, gy, *go, 10, networks.act_params("dense"), seed=int(net),
                                           go_out_per_gr=4, mf_per_go=16, vel=147)
    f = io.BytesIO()
    st.writeState(f)
    return f.getvalue()


@functools.lru_cache(maxsize=None)
def _network(net):
    """The network, loaded once as a user's program holds it."""
    return cbm.CBMState(io.BytesIO(_image(net)))


def _weights(state, rng):
    w = state.array("pfSynWeightPC", 0)
    w[:] = rng.uniform(0.3, 0.7, w.size).astype(np.float32)


def _rates(num_mf, seed):
    bg, cs = networks.eyelid_mf_rates(num_mf, seed)
    return np.stack([bg, cs, cs])


def _stream(num_mf, steps, seed):
    """Eyelid MF input with a CS in the middle."""
    return networks.eyelid_mf_stream(num_mf, steps, seed=seed, cs_on=steps // 3, cs_off=2 * steps // 3, trial_len=steps)


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.Generator(np.random.PCG64([seed, 77]))
    s = {"case": dict(case)}
    if kind in ("loop", "run", "dense"):
        st = _network(case["net"])
        _weights(st, rng)
        if kind == "loop":
            s["mf"] = _stream(st.con("numMF"), case["steps"], seed)
            sim = cbm.CBMSimCore(st, [seed % 1000 + 1])
        else:
            sim = cbm.CBMSimCore(st, [seed % 1000 + 1], resident_steps=500)
            if kind == "run":
                sim.load_mf_stream(cbm.mf_bits(_stream(st.con("numMF"), 500, seed), sim.mf_words()))
            else:
                coding = networks.StateVariableMF(st.con("numMF"), seed=seed)
                sim.set_statevar_input(coding, coding.trajectory(2000), mfSeed=seed % 10000)
        sim.getMZoneList()[0].setGRPCPlastSteps(-0.0005, 0.0005)
        s["sim"] = sim
    elif kind == "session":
        st = _network(str(case["p2"]))
        _weights(st, rng)
        s["state"] = st
        s["sim"] = cbm.CBMSimCore(st, [seed % 1000 + 1])
        s["rates"] = _rates(st.con("numMF"), seed)
        on = case["trial"] // 3
        s["protocol"] = cbm.eyelid_protocol_defaults(
            st, trialSteps=case["trial"], csOn=on, csOff=2 * on, csPhasicOff=on, plastOnDelay=20, plastOffDelay=20,
            preCS=32, postCS=32, binSteps=case["bin"], dataStartTrial=0, numDataTrials=case["trials"],
            mfSeed=seed % 10000)
    elif kind == "sweep":
        params, mf_seeds = sweep.draw_params(case["n"], seed)
        states = []
        for i in range(case["n"]):
            st = cbm.CBMState(io.BytesIO(_image("c1")))
            _weights(st, rng)
            st.setActParam("threshBaseGO", st.act("threshBaseGO") * params[i, 0])
            st.setActParam("gGRIncGO", st.act("gGRIncGO") * params[i, 5])
            states.append(st)
        b = cbm.CBMBatch(states, [[11 + i] for i in range(case["n"])])
        for i, st in enumerate(states):
            proto = cbm.eyelid_protocol_defaults(st, mfSeed=int(mf_seeds[i]) & 0x7FFFFFFF, numDataTrials=3,
                                                 dataStartTrial=0, **sweep.TRIAL)
            proto["plastLTD"] *= params[i, 1]
            proto["plastLTP"] *= params[i, 2]
            b.set_eyelid_protocol(i, sweep.mf_rates(st.con("numMF"), params[i], mf_seeds[i]), **proto)
        s["batch"], s["states"] = b, states
    elif kind == "batch":
        states = [cbm.CBMState(io.BytesIO(_image(p))) for p in case["p2"].split(",")]
        for st in states:
            _weights(st, rng)
            st.setActParam("threshBaseGO", st.act("threshBaseGO") * float(rng.uniform(0.8, 1.2)))
        b = cbm.CBMBatch(states, [[7 + i] for i in range(len(states))])
        for i, st in enumerate(states):
            proto = cbm.eyelid_protocol_defaults(st, trialSteps=400, csOn=100, csOff=200, csPhasicOff=100,
                                                 preCS=100, postCS=100, numDataTrials=3, mfSeed=seed % 10000 + 17 * i)
            proto["plastLTD"] *= float(np.exp(rng.uniform(np.log(0.5), np.log(2.0))))
            b.set_eyelid_protocol(i, _rates(st.con("numMF"), seed + i), **proto)
        s["batch"], s["states"] = b, states
    elif kind == "pfpc":
        n = case["pcs"] * case["fibres"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # spike buffers at a few percent of spikes a step, one delay bit a fibre
        ap = torch.zeros(n, dtype=torch.int32, device="cuda")
        for k in range(32):
            ap |= (torch.rand(n, generator=g, device="cuda") < 0.03).to(torch.int32) << k
        d = torch.randint(1, 9, (n,), generator=g, device="cuda", dtype=torch.int32)
        s["ap"], s["mask"] = ap, torch.ones_like(d) << d
        s["w"] = torch.rand(n, generator=g, device="cuda")
        s["out"] = torch.zeros(case["pcs"], device="cuda")
        fn = cbm.lib.cbm_pfpc_sums_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint32] * 2 + [ctypes.c_void_p] * 2
        s["fn"] = fn
    else:
        x, t, p = _mlp_data(case, seed)
        sizes = [int(v) for v in case["sizes"].split(",")]
        net = MLP(*sizes, max_batch=case["max_batch"], seed=seed % 10000)
        flat = net.get_params()
        for view, src in zip(net.unpack(flat), p):
            view[:] = 0
            view[tuple(slice(0, k) for k in src.shape)] = src
        net.set_params(flat)
        s.update(net=net, x=x, t=t)
    return s


def _mlp_data(case, seed):
    """Feature rows in [-1, 1], log(1 + rate) traces, and He-uniform weights
    with small biases: (x, t, [W1, b1, W2, b2, W3, b3])."""
    n_in, h1, h2, n_out = [int(v) for v in case["sizes"].split(",")]
    rng = np.random.Generator(np.random.PCG64([seed, 5]))
    x = rng.uniform(-1, 1, (case["rows"], n_in)).astype(np.float32)
    t = np.log1p(rng.gamma(1.5, 15.0, (case["rows"], n_out))).astype(np.float32)
    p = []
    for o, i in ((h1, n_in), (h2, h1), (n_out, h2)):
        a = np.sqrt(6.0 / i)
        p += [rng.uniform(-a, a, (o, i)).astype(np.float32), rng.uniform(-0.1, 0.1, o).astype(np.float32)]
    return x, t, p


# ----------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "loop":
        sim = s["sim"]
        zone = sim.getMZoneList()[0]
        nc = []
        for row in s["mf"]:
            sim.updateMFInput(row)
            sim.calcActivity()
            nc.append(zone.exportAPNC())
        return {"nc": np.stack(nc), "vmNC": zone.exportVmNC(), "vmPC": zone.exportVmPC()}
    if kind in ("run", "dense"):
        sim = s["sim"]
        sim.run(case["steps"], case["chunk"])
        zone, innet = sim.getMZoneList()[0], sim.getInputNet()
        out = {"vmNC": zone.exportVmNC(), "vmPC": zone.exportVmPC(), "vmGO": innet.exportVmGO(),
               "apBufNC": zone.exportAPBufNC()}
        if kind == "run":
            out["weights"] = zone.exportPFPCWeights()
            out["vmGR"] = innet.exportVmGR()
        else:
            out["apGR"] = innet.exportAPGR()
        return out
    if kind == "session":
        sim = s["sim"]
        sim.set_eyelid_protocol(s["rates"], **s["protocol"])
        sim.record_gr()
        sim.record_trial_data()
        sim.run(case["trial"] * case["trials"], case["chunk"])
        td = sim.trial_data()
        return {"nc": sim.trial_record("nc"), "pc": sim.trial_record("pc"), "gr": sim.trial_record("gr"),
                "psh": td["psh"], "raster": td["raster"], "eyelid": td["eyelid"]}
    if kind in ("sweep", "batch"):
        b = s["batch"]
        b.run(case["steps"], case["chunk"])
        return {k: np.stack([b.trial_record(i, k) for i in range(len(s["states"]))]) for k in ("nc", "pc", "eyelid")}
    if kind == "forward":
        return s["net"].forward(s["x"])
    if kind == "gradients":
        g, loss = s["net"].gradients(s["x"], s["t"])
        return {"grads": s["net"].unpack(g), "loss": loss}
    if kind == "train":
        net = s["net"]
        loss = net.train(s["x"], s["t"], batch=case["batch"], epochs=1, lr=1e-3, seed=3)
        return {"params": net.unpack(net.get_params()), "loss": loss}
    rc = s["fn"](s["ap"].data_ptr(), s["mask"].data_ptr(), s["w"].data_ptr(), s["ap"].numel(), case["pcs"],
                 s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(cbm.lib.cbm_last_error().decode())
    return s["out"]


# ---------------------------------------------------------------------- work
# Per GR and step: five float state values and the spike buffer read and
# written, the PF delay, the PF->PC weight; every fifth step the history read
# and written and the weight written.  A GR's synapses need be touched only
# when a spike arrives: they are not counted.
STEP_BYTES = 48 + 1 + 4 + (16 + 4) / 5
STEP_FLOPS = 32


def _grs(case):
    if case["kind"] in ("loop", "run", "dense"):
        return {"c1": 1 << 14, "c2": 1 << 20, "c3": 1 << 22}.get(case["net"]) or 1 << int(case["net"])
    if case["kind"] == "session":
        return 1 << case["p2"]
    if case["kind"] == "sweep":
        return case["n"] << 14
    return sum(1 << int(p) for p in case["p2"].split(","))


def work(case):
    kind = case["kind"]
    if kind == "pfpc":
        n = case["pcs"] * case["fibres"]
        return {"bytes": 12 * n + 4 * case["pcs"], "flops": 2 * n}
    if kind in ("forward", "gradients", "train"):
        n_in, h1, h2, n_out = [int(v) for v in case["sizes"].split(",")]
        params = n_in * h1 + h1 * h2 + h2 * n_out + h1 + h2 + n_out
        rows = case["rows"]
        if kind == "forward":
            return {"bytes": 4 * (rows * (n_in + n_out) + params), "flops": 2 * rows * params}
        if kind == "gradients":
            return {"bytes": 4 * (rows * (n_in + n_out) + 2 * params), "flops": 6 * rows * params}
        rows -= rows % case["batch"]
        return {"bytes": 4 * (rows * (n_in + n_out) + 2 * params), "flops": 6 * rows * params}
    gr = _grs(case)
    steps = case["trial"] * case["trials"] if kind == "session" else case["steps"]
    return {"bytes": int(STEP_BYTES * gr * steps), "flops": STEP_FLOPS * gr * steps}


# --------------------------------------------------------------------- exact
def exact(case, seed):
    """Only the float products have a value in more bits: the simulation's
    single-precision steps in their order are its definition."""
    kind = case["kind"]
    if kind == "pfpc":
        s = prepare(case, seed)
        x = s["w"].double() * ((s["ap"] & s["mask"]) != 0)
        return x.reshape(case["pcs"], -1).sum(1)
    if kind not in ("forward", "gradients"):
        return None
    x, t, p = _mlp_data(case, seed)
    x, t = torch.from_numpy(x).double(), torch.from_numpy(t).double()
    p = [torch.from_numpy(v).double().requires_grad_(True) for v in p]
    h = torch.relu(x @ p[0].T + p[1])
    h = torch.relu(h @ p[2].T + p[3])
    y = h @ p[4].T + p[5]
    if kind == "forward":
        return y.detach().numpy()
    loss = ((y - t) ** 2).mean()
    loss.backward()
    pads = [-(-int(v) // 64) * 64 for v in case["sizes"].split(",")]
    grads = []
    for v, shape in zip(p, [(pads[1], pads[0]), (pads[1],), (pads[2], pads[1]), (pads[2],), (pads[3], pads[2]), (pads[3],)]):
        g = np.zeros(shape)
        g[tuple(slice(0, k) for k in v.shape)] = v.grad.numpy()
        grads.append(g)
    return {"grads": grads, "loss": loss.item()}
