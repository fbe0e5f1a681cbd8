"""When a forward may read its weights before the kernel in front of it has finished: only weights that nobody writes any more."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_parity import ALL_DT, assert_matmul_close, dev, make_case  # noqa: E402,F401


def test_first_forward_waits_and_later_ones_do_not(dev, oracle):
    import lloom_b200 as lb
    from lloom_b200 import quantized as Q

    _, x, wq = make_case(oracle, 12, 64, 512, 1, seed=1)
    qt = lb.QTensor.from_data(wq.tobytes(), 12, (64, 512), dev)
    mm, xt = lb.QMatMul.from_qtensor(qt), torch.from_numpy(x).to(dev)
    assert not qt.storage._native.overlaps()  # the upload may be the kernel in front
    mm.forward(xt)
    assert qt.storage._native.overlaps()
    Q.gemm(qt, Q.quantize_act(qt.dtype(), xt), 1)  # the package's own entries only read
    Q.gemv(qt, Q.quantize_act(qt.dtype(), xt), 1)
    assert qt.storage._native.overlaps()
    qt.device_ptr()  # its holder may write through it
    assert not qt.storage._native.overlaps()
    mm.forward(xt)
    assert not qt.storage._native.overlaps()


@pytest.mark.parametrize("how", ["pointer", "tensor"])
@pytest.mark.parametrize("dt", ALL_DT)
def test_blocks_rewritten_by_the_kernel_in_front(dev, oracle, dt, how):
    """A holder of the device pointer, or of the tensor a storage was made over, rewrites the blocks by a kernel directly in
    front of a forward: the forward uses the new ones."""
    import lloom_b200 as lb

    n, k = 4096, 1024
    _, x, wa = make_case(oracle, dt, n, k, 1, seed=dt)
    _, _, wb = make_case(oracle, dt, n, k, 1, seed=dt + 1)
    if how == "pointer":
        st = lb.QCudaStorage.load_quantized(dev, wa.tobytes(), lb.GgmlDType(dt))
        st.device_ptr()
        buf = st._data
    else:
        buf = torch.from_numpy(np.concatenate([wa.reshape(-1), np.zeros(1024, np.uint8)])).to(dev)
        st = lb.QCudaStorage(buf, wa.size, lb.GgmlDType(dt))
    mm = lb.QMatMul.from_qtensor(lb.QTensor(st, (n, k)))
    xt = torch.from_numpy(x).to(dev)
    new = [torch.from_numpy(w.reshape(-1)).to(dev) for w in (wa, wb)]
    sample = np.arange(0, n, 7)
    want = [(oracle.matmul(dt, x, w[sample], len(sample)), oracle.matmul_absum(dt, x, w[sample], len(sample))) for w in (wa, wb)]
    mm.forward(xt)
    for turn in (1, 0, 1):
        torch.bitwise_xor(new[turn], 0, out=buf[:wa.size])  # a kernel, not a copy
        got = mm.forward(xt)
        assert not st._native.overlaps()
        assert_matmul_close(got.cpu().numpy()[:, sample], *want[turn], f"turn {turn}")


@pytest.mark.parametrize("dt", ALL_DT)
@pytest.mark.parametrize("m,k", [(1, 1024), (5, 1024), (40, 1024), (200, 1024), (3, 4096), (5, 4096), (1, 11264)])
def test_switch_decides_for_every_storage(dev, oracle, dt, m, k):
    """On and off hold whether or not the storage's pointer has been handed out; without either the storage decides.  The
    bits are the same in all six."""
    import lloom_b200 as lb
    from lloom_b200 import _lib

    n = 1030
    _, x, wq = make_case(oracle, dt, n, k, m, seed=m)
    xt = torch.from_numpy(x).to(dev)
    qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
    mm = lb.QMatMul.from_qtensor(qt)
    want = mm.forward(xt)
    start = _lib.lib().lloom_b200_set_launch_overlap(-1)
    try:
        for exposed in (False, True):
            if exposed:
                qt.device_ptr()
            for mode, early in ((1, True), (0, False), (-1, not exposed)):
                _lib.lib().lloom_b200_set_launch_overlap(mode)
                assert qt.storage._native.overlaps() == early, (exposed, mode)
                for _ in range(3):
                    assert torch.equal(mm.forward(xt), want)
    finally:
        _lib.lib().lloom_b200_set_launch_overlap(start)
