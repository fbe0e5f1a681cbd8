"""Calls past the limits of one launch: more routed products, or more groups of activation rows, than a
grid dimension holds; and calls with the least workspace an entry asks for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_parity import ALL_DT, dev, make_case  # noqa: E402,F401


@pytest.mark.parametrize("in_dim1", [1, "topk"])
def test_experts_past_one_grid(dev, oracle, in_dim1):
    """70000 experts per token, two tokens: three launches, two of which start or end in the middle of a token.  Every
    product has the bits of the expert's own forward."""
    import lloom_b200 as lb

    n_experts, n, k, topk, batch = 5, 3, 256, 70000, 2
    _, _, wq = make_case(oracle, 12, n_experts * n, k, 1, seed=11)
    gen = torch.Generator(device=dev).manual_seed(1)
    ids = torch.randint(0, n_experts, (batch, topk), generator=gen, device=dev)
    rows = 1 if in_dim1 == 1 else topk
    x = torch.randn(batch, rows, k, generator=gen, device=dev)
    got = lb.QTensor.from_data(wq.tobytes(), 12, (n_experts, n, k), dev).indexed_moe_forward(x, ids)
    assert tuple(got.shape) == (batch, topk, n)
    every = lb.QMatMul.from_qtensor(lb.QTensor.from_data(wq.tobytes(), 12, (n_experts * n, k), dev))
    check = np.r_[0:3, 61068:61073, 65533:65538, topk - 3:topk]  # the ends of the tokens and of the launches
    for b in range(batch):
        for t in (check if rows > 1 else [0]):
            y = every.forward(x[b, t:t + 1]).view(n_experts, n)
            want, have = (y[ids[b]], got[b]) if rows == 1 else (y[ids[b, t]], got[b, t])
            assert torch.equal(have, want), (b, t)


def test_activation_rows_past_one_grid(dev, oracle):
    """Shapes without a tcgen05 GEMM take any number of activation rows through the skinny kernel, 48 to a group: 65535 groups
    and five rows more, from values and from canonical blocks.  Rows on both sides of the edge have the bits they have in a
    call of their own (k = 64 is one superblock: its sum is not split)."""
    import lloom_b200 as lb
    from lloom_b200 import quantized as Q

    n, k, m = 2, 64, 65535 * 48 + 5
    _, _, wq = make_case(oracle, 8, n, k, 1, seed=12)
    qt = lb.QTensor.from_data(wq.tobytes(), 8, (n, k), dev)
    mm = lb.QMatMul.from_qtensor(qt)
    x = torch.randn(m, k, generator=torch.Generator(device=dev).manual_seed(2), device=dev, dtype=torch.float16)
    spans = [(0, 100), (m - 105, m)]
    got = mm.forward(x)
    for a, b in spans:
        assert torch.equal(got[a:b], mm.forward(x[a:b].clone()))
    del x, got
    blocks = Q.quantize_act(lb.GgmlDType.Q8_0, torch.randn(m, k, device=dev))
    got = Q.gemm(qt, blocks, m)
    for a, b in spans:
        assert torch.equal(got[a:b], Q.gemm(qt, blocks[a:b].clone(), b - a))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt,k", [(12, 512), (14, 14336), (8, 192), (2, 4096)])
@pytest.mark.parametrize("m", [1, 3, 8])
def test_gemm_of_a_decode_batch_needs_no_workspace(dev, oracle, dt, k, m):
    """lloom_b200_gemm with up to eight rows of canonical blocks: the GEMV's bits, no workspace."""
    import lloom_b200 as lb
    from lloom_b200 import _lib
    from lloom_b200 import quantized as Q

    n = 40
    _, x, wq = make_case(oracle, dt, n, k, m, seed=m)
    qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
    act = Q.quantize_act(lb.GgmlDType(dt), torch.from_numpy(x).to(dev))
    y = torch.empty(m, n, device=dev)
    rc = _lib.lib().lloom_b200_gemm(dt, qt.storage._ptr(), act.data_ptr(), y.data_ptr(), m, n, k, n, None, 0,
                                    torch.cuda.current_stream(dev).cuda_stream)
    assert rc == _lib.OK and torch.equal(y, Q.gemv(qt, act, m))


@pytest.mark.parametrize("dt", ALL_DT)
@pytest.mark.parametrize("m", [1, 3, 8, 40, 128, 130])
def test_forward_keeps_to_its_workspace(dev, oracle, dt, m):
    """A workspace of exactly the size asked for, with a strip behind it that no forward may touch."""
    import lloom_b200 as lb
    from lloom_b200 import _lib

    L, n = _lib.lib(), 300
    for k in (512, 11264):
        _, x, wq = make_case(oracle, dt, n, k, m, seed=m)
        qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
        xt = torch.from_numpy(x).to(dev)
        need = int(L.lloom_b200_workspace_bytes(dt, m, n, k))
        ws = torch.full((need + 4096,), 0xA5, dtype=torch.uint8, device=dev)
        y = torch.empty(m, n, device=dev)
        stream = torch.cuda.current_stream(dev).cuda_stream
        args = (dt, qt.storage._ptr(), xt.data_ptr(), y.data_ptr(), m, n, k, n, ws.data_ptr())
        assert L.lloom_b200_qmatmul_fwd(*args, need, stream) == _lib.OK
        assert torch.equal(y, lb.QMatMul.from_qtensor(qt).forward(xt))
        assert bool((ws[need:] == 0xA5).all())
        assert L.lloom_b200_qmatmul_fwd(*args, need - 1, stream) == _lib.ERR_WORKSPACE
