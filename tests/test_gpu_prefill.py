"""Prefill GEMMs (more than 128 activation rows) where the operand images can go wrong: a last weight tile of one row or all
but one, an odd number of tiles, the shortest rows, activation tiles of one row and of all but one; and the prebuilt
image against the one a call builds itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_parity import ALL_DT, assert_matmul_close, dev, make_case, run_fwd  # noqa: E402,F401
from test_gpu_skinny import check  # noqa: E402

SHORT = {8: 128, 2: 128, 6: 128, 12: 256, 13: 256, 14: 256}  # shortest row of a GEMM: a pipeline stage, a superblock


@pytest.mark.parametrize("dt", ALL_DT)
@pytest.mark.parametrize("n", [1, 127, 129, 300])
def test_edges(dev, oracle, dt, n):
    for k, m in ((SHORT[dt], 129), (3 * SHORT[dt], 255), (1280, 257)):
        check(dev, oracle, dt, n, k, m, seed=n)


@pytest.mark.parametrize("dt", ALL_DT)
def test_prebuilt_image(dev, oracle, dt):
    import lloom_b200 as lb

    n, k, m = 200, 768, 140
    _, x, wq = make_case(oracle, dt, n, k, m, seed=4)
    qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
    qt.storage.build_prefill_image(qt.shape)
    got = lb.QMatMul.from_qtensor(qt).forward(torch.from_numpy(x).to(dev)).cpu().numpy()
    assert got.tobytes() == np.asarray(run_fwd(dev, dt, wq, n, k, x)).tobytes()


@pytest.mark.parametrize("dt,n,stays,m", [(12, 12288, 48, 49), (13, 5120, 64, 65), (13, 3072, 96, 128), (14, 12300, 48, 64), (14, 5121, 64, 65),
                                          (14, 3073, 96, 97), (8, 10240, 96, 97), (2, 10241, 96, 128), (6, 10240, 96, 121)])
def test_short_prompts_with_an_image(dev, oracle, dt, n, stays, m):
    """Where an image moves a prompt of up to 128 rows to the GEMM: the bits of that kernel, and the oracle's values on
    sampled columns.  With `stays` rows it is the packed blocks' kernel, with or without the image."""
    import lloom_b200 as lb

    k = 2048
    _, x, wq = make_case(oracle, dt, n, k, m, seed=m)
    qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
    mm, xt = lb.QMatMul.from_qtensor(qt), torch.from_numpy(x).to(dev)
    long = torch.cat([xt, torch.zeros(200 - m, k, device=dev)])  # past 128 rows: the GEMM, whatever the matrix
    gemm, packed = mm.forward(long)[:m], mm.forward(xt)
    assert qt.storage.build_prefill_image(qt.shape)
    got = mm.forward(xt)
    assert torch.equal(got, gemm) and not torch.equal(got, packed)
    short = mm.forward(xt[:stays])
    sub = np.arange(0, n, 37)
    wsub = np.ascontiguousarray(wq[sub])
    ref = oracle.matmul(dt, x, wsub, len(sub), nthreads=8)
    assert_matmul_close(got.cpu().numpy()[:, sub], ref, oracle.matmul_absum(dt, x, wsub, len(sub), nthreads=8), f"n={n} m={m}")
    qt.storage.drop_prefill_image()
    assert torch.equal(short, mm.forward(xt[:stays]))


@pytest.mark.parametrize("dt", [12, 8])
def test_short_rows_ignore_an_image(dev, oracle, dt):
    """Rows of fewer than 2048 elements stay with the packed blocks up to 128 activation rows."""
    import lloom_b200 as lb

    n, k, m = 12288, 1792, 128
    _, x, wq = make_case(oracle, dt, n, k, m, seed=3)
    qt = lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev)
    mm, xt = lb.QMatMul.from_qtensor(qt), torch.from_numpy(x).to(dev)
    packed = mm.forward(xt)
    assert qt.storage.build_prefill_image(qt.shape)
    assert torch.equal(mm.forward(xt), packed)


def test_image_of_several_slabs(dev, oracle):
    """A matrix whose image is past the slab limit is expanded and multiplied in parts: rows of both parts against the oracle,
    and the bits of the prebuilt image, which is read in one."""
    import lloom_b200 as lb

    n, k, m = 20000, 4096, 129  # 128 tiles of weight rows to a slab of 256 MB: 16384 rows and the rest
    _, x, base = make_case(oracle, 14, 512, k, m, seed=8)
    wq = base[np.random.default_rng(9).integers(0, 512, n)]
    qt = lb.QTensor.from_data(wq.tobytes(), 14, (n, k), dev)
    mm, xt = lb.QMatMul.from_qtensor(qt), torch.from_numpy(x).to(dev)
    got = mm.forward(xt)
    sub = np.r_[0:40, 16344:16424, n - 40:n]
    ref = oracle.matmul(14, x, np.ascontiguousarray(wq[sub]), len(sub), nthreads=8)
    absum = oracle.matmul_absum(14, x, np.ascontiguousarray(wq[sub]), len(sub), nthreads=8)
    assert_matmul_close(got.cpu().numpy()[:, sub], ref, absum, "slabs")
    assert qt.storage.build_prefill_image(qt.shape)
    assert torch.equal(mm.forward(xt), got)


def test_q6k_tile_shapes(dev, oracle):
    """Few tiles take 128-row ones, many 256-row ones: a row has the same bits in both."""
    n, k = 9600, 256  # 75 tiles of weight rows: 150 small or 75 large ones for 256 activation rows
    _, x, wq = make_case(oracle, 14, n, k, 256, seed=5)
    large = np.asarray(run_fwd(dev, 14, wq, n, k, x))
    small = np.asarray(run_fwd(dev, 14, wq.reshape(-1)[:4096 * 210], 4096, k, x))
    assert np.ascontiguousarray(large[:, :4096]).tobytes() == small.tobytes()
