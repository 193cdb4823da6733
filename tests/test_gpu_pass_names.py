"""CBM_PASS_TMA takes the geometries it names and refuses the others: unknown tuples,
slot bounds below the network's slots and more rows than a tile has; the geometry
in use reports the pipeline that runs."""
import pytest

pytestmark = pytest.mark.gpu

SMALL, WIDE = ((7, 7, 4, 4, 9), dict(mf_per_gr=4)), ((9, 8, 4, 4, 9), dict(mf_per_gr=5))


@pytest.mark.parametrize("net,name,reported", [
    (WIDE, "4,1,4,1,0", (4, 16, 4)), (WIDE, "8,1,3,2,0", (8, 32, 3)), (WIDE, "2,1,4,1,0", (2, 8, 4)),
    (WIDE, "4,1,2,4,0", (4, 16, 2)), (WIDE, "1,1,4,1,0", (1, 4, 4)), (SMALL, "2,1,4,1,0", (2, 8, 4)),
    (WIDE, "4,2,2,4,4", "more synapse slots"), (WIDE, "4,1,4,4,4", "more synapse slots"),
    (WIDE, "4,1,4,3,0", "not compiled in"), (WIDE, "5,1,4,4,0", "not compiled in"), (WIDE, "4,3,2,4,0", "not compiled in"),
    (SMALL, "8,1,3,2,0", "more rows per stage"), (SMALL, "4,2,2,4,4", "more rows per stage"), (WIDE, "4,1,4", "must be"),
])
def test_named_geometry(net, name, reported, monkeypatch):
    import cerebellum_simulation_b200 as cbm
    from cerebellum_simulation_b200 import networks
    dims, opt = net

    def new_state(con, *args, **kw):
        con = con.replace("maxnumpGRfromGOtoGR 4", "maxnumpGRfromGOtoGR 5")
        return cbm.CBMState.new(con.replace("maxnumpGRfromMFtoGR 4", "maxnumpGRfromMFtoGR 5"), *args, **kw)

    st = networks.build_random_network(*dims, networks.act_params("dense"), seed=2, go_out_per_gr=4, mf_per_go=8, vel=60,
                                       new_state=new_state, **opt)
    monkeypatch.setenv("CBM_PASS_TMA", name)
    if isinstance(reported, str):
        with pytest.raises(cbm.CBMError, match=reported):
            cbm.CBMSimCore(st, [3], device=0)
        return
    sim = cbm.CBMSimCore(st, [3], device=0)
    assert tuple(sim.pass_geometry()) == ("grPassTmaKernel", *reported)
    sim.close()
