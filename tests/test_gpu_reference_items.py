"""The reference energy call at the edges of its item split: structures of less
than a chunk of 32 beads, whole tiles, a bead more, and both sides of the size
where chunks give way to whole tiles; all three entry points against the FP64
oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_RTOL = 1e-5  # FP32 pair terms, FP64 sums: the bound of the other energy tests


def _system(n_beads, seed):
    """Two chains and crowders on a jittered lattice, n_beads in all."""
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.model import CROWDER_TYPE, Molecule, System
    rng = np.random.default_rng(seed)
    lengths = [min(12, n_beads // 2), min(17, n_beads - n_beads // 2)]
    crowders = n_beads - sum(lengths)
    k = int(np.ceil((crowders + 64) ** (1 / 3))) + 2
    box = 13.0 * k
    table = synth.contact_table(rng)
    s = synth.build_system(rng, table, lengths, 0, 0.0, box)
    grid = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * 13.0 + 6.5
    beads = np.concatenate([m.pos for m in s.molecules])
    d = grid[:, None] - beads[None]
    d -= box * np.round(d / box)
    grid = grid[(d ** 2).sum(-1).min(1) > 64.0][:crowders] + rng.uniform(-1, 1, size=(crowders, 3))
    mols = list(s.molecules)
    for c in grid:
        m = Molecule.from_beads([CROWDER_TYPE], np.zeros((1, 3), np.float32))
        m.crowder = True
        m.set_position(c.astype(np.float32))
        mols.append(m)
    return System(mols, s.box, table, crowder_radius=6.0)


@pytest.mark.parametrize("n_beads", [2, 29, 31, 128, 129, 1300, 6144, 6145])
def test_reference_call_sizes(built_lib, n_beads):
    import torch
    from oracle import bindings as ob
    from remcdockingsimulator_b200.engine import make_params
    from remcdockingsimulator_b200.reference_abi import abi, pack_reference_layout
    s = _system(n_beads, n_beads)
    assert s.n_beads == n_beads
    want = ob.FP64Oracle(s, make_params()).energy(s.state()[0])
    L, p = abi(), C.c_void_p
    pos, meta = pack_reference_layout(s, 32)
    P = pos.shape[0]
    dp, dm = torch.from_numpy(pos).cuda(), torch.from_numpy(meta).cuda()
    dt = torch.from_numpy(np.ascontiguousarray(s.table.pairs, np.float32)).cuda()
    L.CUDA_setBoxDimension(s.box)
    sync = C.c_double(0.0)
    for _ in range(2):  # the finished-items counter is back at zero for the second
        L.CUDA_EonDevice(p(dp.data_ptr()), p(dm.data_ptr()), None, None, None, p(dt.data_ptr()),
                         C.byref(sync), 32, P, 0)
        assert L.remc_reference_abi_status() == 0
        assert abs(sync.value - want) <= E_RTOL * max(abs(want), 1e-3)
    g = P // 32
    grid = torch.full((g * g,), 7.0, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    L.CUDA_EonDevice_async(p(dp.data_ptr()), p(dm.data_ptr()), None, None, None, p(dt.data_ptr()),
                           p(grid.data_ptr()), g, 32, P, 0, p(stream.cuda_stream))
    stream.synchronize()
    kbt = float(make_params().kbt_cf)
    assert abs(grid.double().sum().item() * kbt - sync.value) <= 1e-6 * max(abs(sync.value), 1e-3)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    assert L.CUDA_EonDevice_noalloc(p(dp.data_ptr()), p(dm.data_ptr()), p(dt.data_ptr()), P,
                                    p(out.data_ptr()), p(torch.cuda.current_stream().cuda_stream)) == 0
    assert abs(out.item() - sync.value) <= 1e-12 * abs(sync.value)


@pytest.mark.parametrize("ti,tj,entry", [
    (3.0, 7.0, 67), (19.0, 19.0, 399), (float("nan"), 4.0, 0), (2.0, float("nan"), 0),
    (-3.0, 4.0, 0), (-2e7, 4.0, 0), (25.0, 0.0, 399), (2e9, 0.0, 399), (float("inf"), 0.0, 399),
    (float("-inf"), 5.0, 0), (1.0, 0.4, 20), (1.0, 0.6, 21),
])
def test_contact_table_entry(built_lib, ti, tj, entry):
    """The entry of a pair is the nearest of 20 ti + tj in the table, the first
    one where that is no number: a table of zeros but for it gives the energy
    that a table of that value throughout gives."""
    import torch
    from remcdockingsimulator_b200.reference_abi import abi
    L, p = abi(), C.c_void_p
    pos = torch.tensor([[10.0, 10.0, 10.0, 0.0], [15.0, 10.0, 10.0, 1.0]], device="cuda")
    meta = torch.tensor([[ti, 0.0, 6.0, 0.0], [tj, 0.0, 6.0, 0.0]], device="cuda")
    L.CUDA_setBoxDimension(100.0)

    def energy(table):
        out = C.c_double(0.0)
        L.CUDA_EonDevice(p(pos.data_ptr()), p(meta.data_ptr()), None, None, None,
                         p(table.data_ptr()), C.byref(out), 32, 2, 0)
        assert L.remc_reference_abi_status() == 0
        return out.value

    one = torch.zeros(400, device="cuda")
    one[entry] = -5.0
    torch.cuda.synchronize()
    want = energy(torch.full((400,), -5.0, device="cuda"))
    assert energy(one) == want and want != energy(torch.zeros(400, device="cuda"))
