"""The tensor-core skinny kernel (2 to 128 activation rows, single rows against long weight rows, shapes the tcgen05 GEMMs do
not take) and the typed forward, at the sizes where they can go wrong: edges of the 8-row activation tiles and of their
groups, of 16-row weight tiles and CTA ranges, superblocks that do not fill the slots, rows that end in the middle of a
superblock or start off 16-byte boundaries."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_parity import ALL_DT, DT_NAMES, assert_matmul_close, dev, make_case, run_fwd  # noqa: E402,F401


def check(dev, oracle, dt, n, k, m, seed=1):
    _, x, wq = make_case(oracle, dt, n, k, m, seed=seed)
    got = run_fwd(dev, dt, wq, n, k, x)
    ref = oracle.matmul(dt, x, wq, n, nthreads=8)
    assert_matmul_close(got, ref, oracle.matmul_absum(dt, x, wq, n, nthreads=8), f"{DT_NAMES[dt]} n={n} k={k} m={m}")


@pytest.mark.parametrize("dt", ALL_DT)
@pytest.mark.parametrize("m", [2, 7, 9, 16, 17, 24, 25, 33, 48, 49, 97, 128])
def test_activation_tiles(dev, oracle, dt, m):
    """One tile to several groups of tiles, with and without a ragged last one; one superblock to more than the slots."""
    for n, k in ((33, 256), (17, 768), (50, 2560)):
        check(dev, oracle, dt, n, k, m, seed=m)


@pytest.mark.parametrize("dt", [8, 2, 6])
@pytest.mark.parametrize("k", [64, 192, 320, 576, 2112])
def test_rows_not_whole_superblocks(dev, oracle, dt, k):
    """32-element formats end a row after any multiple of 64; such rows start anywhere modulo 16 bytes."""
    for n, m in ((1, 2), (16, 8), (35, 130)):
        check(dev, oracle, dt, n, k, m, seed=k)


@pytest.mark.parametrize("dt", ALL_DT)
def test_row_ranges(dev, oracle, dt):
    """A last tile of one row, CTA ranges of one and two tiles, more tiles than one round of warps."""
    for n in (1, 15, 16, 2369, 7600):
        check(dev, oracle, dt, n, 512, 5, seed=n)


@pytest.mark.parametrize("dt", [12, 13])
@pytest.mark.parametrize("m", [2, 5, 8])
def test_two_sums_per_warp(dev, oracle, dt, m):
    """Three or more weight tiles per CTA: a warp keeps the sums of two slots.  Superblocks that fill a slice of eight, one more,
    and five and thirteen, so that some second slots stay empty; a last tile of one row.  Same bits as the rows alone and as
    a row shard with fewer tiles, where neither does."""
    n = 16 * 148 * 2 + 33
    for k in (1280, 2048, 2304, 3328):
        _, x, wq = make_case(oracle, dt, n, k, m, seed=k)
        got = np.asarray(run_fwd(dev, dt, wq, n, k, x))
        alone = np.concatenate([run_fwd(dev, dt, wq, n, k, x[r:r + 1]) for r in range(m)])
        assert alone.tobytes() == got.tobytes(), k
        shard = np.asarray(run_fwd(dev, dt, np.ascontiguousarray(wq[-700:]), 700, k, x))
        assert shard.tobytes() == np.ascontiguousarray(got[:, -700:]).tobytes(), k
        sub = np.arange(0, n, 31)
        ref = oracle.matmul(dt, x, np.ascontiguousarray(wq[sub]), len(sub), nthreads=8)
        assert_matmul_close(got[:, sub], ref, oracle.matmul_absum(dt, x, np.ascontiguousarray(wq[sub]), len(sub), nthreads=8), f"k={k}")


@pytest.mark.parametrize("dt", ALL_DT)
def test_single_row_against_long_rows(dev, oracle, dt):
    """k past the dp4a kernel's range: same bits as the row in a batch."""
    n, k = 40, 11264
    _, x, wq = make_case(oracle, dt, n, k, 3, seed=2)
    batch = run_fwd(dev, dt, wq, n, k, x)
    alone = np.concatenate([run_fwd(dev, dt, wq, n, k, x[r:r + 1]) for r in range(3)])
    assert alone.tobytes() == batch.tobytes()
    ref = oracle.matmul(dt, x, wq, n, nthreads=8)
    assert_matmul_close(batch, ref, oracle.matmul_absum(dt, x, wq, n, nthreads=8), DT_NAMES[dt])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 5, 40, 200])
@pytest.mark.parametrize("dt", ALL_DT)
def test_half_precision_in_and_out(dev, oracle, dt, m, dtype):
    """Halves widen exactly before they are quantized and outputs are the f32 results rounded: bit for bit the forward of
    the widened input, cast.  Also from a view that starts off the kernels' 16-byte alignment."""
    import lloom_b200 as lb

    n, k = 70, 1024
    _, x, wq = make_case(oracle, dt, n, k, m, seed=m)
    mm = lb.QMatMul.from_qtensor(lb.QTensor.from_data(wq.tobytes(), dt, (n, k), dev))
    xh = torch.from_numpy(x).to(dev, dtype)
    want = mm.forward(xh.float()).to(dtype)
    got = mm.forward(xh)
    assert got.dtype == dtype and torch.equal(got.view(torch.int16), want.view(torch.int16))
    off = torch.empty(m * k + 1, dtype=dtype, device=dev)[1:].view(m, k).copy_(xh)
    assert torch.equal(mm.forward(off).view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 5])
def test_store_block_of_half_precision(dev, oracle, m, dtype):
    """The storage-level entry with a SiLU on the store returns the input's type, the f32 result cast."""
    import lloom_b200 as lb

    n, k = 70, 1024
    _, x, wq = make_case(oracle, 12, n, k, m, seed=m)
    st = lb.QTensor.from_data(wq.tobytes(), 12, (n, k), dev).storage
    xh = torch.from_numpy(x).to(dev, dtype)
    want = st.fwd((n, k), xh.float(), store=1)
    got = st.fwd((n, k), xh, store=1)
    assert want.dtype == torch.float32 and got.dtype == dtype and torch.equal(got, want.to(dtype))
    out = torch.empty(m, n, device=dev)  # a caller's buffer is f32
    assert st.fwd((n, k), xh, out=out, store=1) is out and torch.equal(out, want)


@pytest.mark.parametrize("ids_dtype", [torch.int64, torch.int32, torch.uint8])
def test_id_types(dev, oracle, ids_dtype):
    import lloom_b200 as lb

    _, x, wq = make_case(oracle, 12, 64, 512, 2, seed=3)
    qt = lb.QTensor.from_data(wq.tobytes(), 12, (64, 512), dev)
    ids = torch.tensor([[5, 63, 0], [7, 7, 31]], device=dev)
    assert torch.equal(qt.embedding(ids.to(ids_dtype)), qt.dequantize()[ids])
    stacked = lb.QTensor.from_data(wq.tobytes(), 12, (4, 16, 512), dev)
    xs = torch.from_numpy(x).to(dev).view(2, 1, 512)
    eids = torch.tensor([[3, 1], [0, 2]], device=dev)
    assert torch.equal(stacked.indexed_moe_forward(xs, eids.to(ids_dtype)), stacked.indexed_moe_forward(xs, eids))
