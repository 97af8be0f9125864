"""The reference energy call on cudaStreamPerThread: one handle value, another
stream in every host thread. Calls of two threads overlap on the GPU, and each
gets its own structure's energy; calls of unlike sizes take turns on a stream."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


def _devices(sizes):
    import torch
    from conftest import crowder_lattice
    from remcdockingsimulator_b200.reference_abi import abi, pack_reference_layout
    out = []
    for k, n in enumerate(sizes):
        s = crowder_lattice(n, seed=30 + k, side=19)
        pos, meta = pack_reference_layout(s, 32)
        table = np.ascontiguousarray(s.table.pairs, np.float32).reshape(-1)
        out.append(tuple(torch.from_numpy(a).cuda() for a in (pos, meta, table)) + (pos.shape[0],))
    abi().CUDA_setBoxDimension(s.box)
    torch.cuda.synchronize()
    return out


def _call(d, res, stream):
    from remcdockingsimulator_b200.reference_abi import abi
    p = C.c_void_p
    abi().CUDA_EonDevice_async(p(d[0].data_ptr()), p(d[1].data_ptr()), None, None, None,
                               p(d[2].data_ptr()), p(res.data_ptr()), 1, 32, d[3], 0, p(stream))
    assert abi().remc_reference_abi_status() == 0


def test_per_thread_streams(built_lib):
    import torch
    dev = _devices([1500, 6800])
    res = [torch.zeros((60, 1), device="cuda") for _ in dev]
    alone = []
    for d in dev:
        r = torch.zeros(1, device="cuda")
        torch.cuda.synchronize()
        _call(d, r, 0)
        torch.cuda.synchronize()
        alone.append(r.item())
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            torch.cuda.set_device(0)
            for i in range(60):
                _call(dev[k], res[k][i], PER_THREAD)
            torch.cuda.ExternalStream(PER_THREAD).synchronize()
        except Exception as e:
            errors.append(e)

    for _ in range(3):  # later threads take over the buffers of ended ones
        for r in res:
            r.zero_()
        torch.cuda.synchronize()
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not errors, errors
        for k in range(2):  # the same FP32 and FP64 sums in the same order
            assert np.all(res[k].cpu().numpy() == np.float32(alone[k])), k


def test_unlike_sizes_on_one_stream(built_lib):
    """Every size's counter of finished items is at zero again after its call."""
    import torch
    dev = _devices([40, 1500, 6143, 6144, 6145, 6800])
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    res = torch.zeros((4, len(dev), 1), device="cuda")
    torch.cuda.synchronize()
    order = [0, 1, 2, 3, 4, 5], [5, 4, 3, 2, 1, 0], [1, 4, 0, 5, 2, 3], [3, 0, 5, 1, 4, 2]
    for i, ks in enumerate(order):
        for k in ks:
            _call(dev[k], res[i, k], stream.cuda_stream)
    torch.cuda.synchronize()
    got = res.cpu().numpy()
    assert np.all(got == got[0]) and np.all(got[0] != 0.0)
    per_thread = torch.zeros((len(dev), 1), device="cuda")
    torch.cuda.synchronize()
    for k in range(len(dev)):
        _call(dev[k], per_thread[k], PER_THREAD)
    torch.cuda.synchronize()
    assert np.all(per_thread.cpu().numpy() == got[0])
