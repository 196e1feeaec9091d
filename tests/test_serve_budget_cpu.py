"""A pool mesh's device bytes, which the server holds against its budget, are those of the
arrays that its arena keeps: one copy of every array, to the byte."""
import pytest


@pytest.mark.parametrize("n,vpb", [(5, 64), (9, 64), (9, 16), (13, 32)])
def test_device_bytes_of_a_3d_mesh(eik, mg, n, vpb):
    xyz, tets = mg.kuhn_cube(n, 0.2, seed=n)
    e = eik.Eikonal(False)
    e.set_mesh(xyz, tets)
    e.deviceSetup_ = 0
    e.maxVertsPerBlock_ = vpb
    e.prepare()
    s, (lab, nb) = e.stats(), e.getPartition()
    b, pairs = lab[tets], set()
    for i in range(4):
        for j in range(4):
            apart = b[:, i] != b[:, j]
            pairs |= set(zip(b[apart, i].tolist(), b[apart, j].tolist()))
    slots, halo, nv = s["total_slots"], round(s["mean_halo_per_block"] * nb), xyz.shape[0]
    layout = nb * 32 + slots * (6 * 4 + 8 + 4) + halo * 4 + (nb + 1 + len(pairs)) * 4
    bounds_and_memos = slots * (8 + 2 * 16)
    # five arrays of times and two of ids a vertex; nine words and a byte a block; seven an instance
    state = nv * 7 * 4 + nb * (9 * 4 + 1) + 7 * 4
    srv = eik.EikonalServer(hbm_budget_bytes=1 << 26)
    info = srv.mesh_info(srv.add_mesh(e))
    srv.close()
    assert info["device_bytes"] == layout + bounds_and_memos + state
