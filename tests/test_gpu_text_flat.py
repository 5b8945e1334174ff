"""The flat lower-triangular text writer around its steps: entry counts around
one and several steps of 512 entries, every type, inputs and texts at any
alignment."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


# n(n-1)/2 entries: 496, 528, 1,035, 2,016, 2,080, 4,095, 4,186, ...
@pytest.mark.parametrize("n", [2, 3, 32, 33, 46, 64, 65, 91, 92, 700])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32])
@pytest.mark.parametrize("skew", [0, 1, 7])
def test_text_at_any_alignment(ctx, n, dtype, skew):
    rng = np.random.default_rng(n)
    e = n * (n - 1) // 2
    top = np.iinfo(dtype).max
    # every number of digits, and the values around each power of ten
    edge = np.array([v for k in range(10) for v in (10**k - 1, 10**k) if v <= top] + [top])
    lt = np.where(rng.random(e) < 0.5, rng.choice(edge, e),
                  (rng.random(e) ** 6 * top)).astype(dtype)
    want = "".join(",".join(map(str, lt[i * (i - 1) // 2:i * (i + 1) // 2])) + "\n"
                   for i in range(1, n)).encode()
    raw = torch.zeros(e * dtype().itemsize + 64, dtype=torch.uint8, device="cuda:0")
    off = skew * dtype().itemsize
    raw[off:off + e * dtype().itemsize] = torch.from_numpy(lt.view(np.uint8).copy())
    text = torch.full((len(want) + 64,), 255, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    nb = ctx.lower_triangular_text_noalloc(raw.data_ptr() + off, n, dtype,
                                           text.data_ptr() + skew, len(want))
    got = text.cpu().numpy()
    assert nb == len(want) and got[skew:skew + nb].tobytes() == want
    assert (got[:skew] == 255).all() and (got[skew + nb:] == 255).all()  # nothing outside
