"""The exact sequential binary32 sum is formed from chunk records of the binades
the running sum is expected in: at the edges of chunks, groups and passes, and for
sums that grow, shrink, cancel, cross zero, jump over many binades or stand on
rounding ties, it equals the sum added term by term, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 511, 512, 513, 4095, 4096, 4097, 131071, 131072, 131073, 700001]


def make(kind, n):
    rng = np.random.default_rng(n)
    v = rng.uniform(0.5, 2.0, n)
    if kind == "signs":
        v = rng.normal(size=n)
    elif kind == "cancel":
        v = np.where(np.arange(n) < n // 2, 1.0, -1.0) * np.where(np.arange(n) % 7 == 0, 1.5, 0.25)
    elif kind == "same":
        v = np.full(n, 1.7320508)
    elif kind == "ties":
        v = rng.choice([0.5, 1.0, 1.5, 2.0 ** -20], n)
    elif kind == "wide":
        v = rng.normal(size=n) * 10.0 ** rng.uniform(-20, 20, n)
    elif kind == "jump":
        v[n // 2:] *= 1.0e6
        v[3 * n // 4:] *= -1.0
    elif kind == "huge":
        v = rng.uniform(-1.0, 1.0, n) * 1.0e32
    elif kind == "zeros":
        v[: 2 * n // 3] = 0.0
    return v.astype(np.float32)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["grow", "signs", "cancel", "same", "ties", "wide", "jump", "huge", "zeros"])
def test_sum_is_the_sequential_one(ctx, kind, n):
    v = make(kind, n)
    want = np.add.accumulate(v, dtype=np.float32)[-1]
    got = ctx.sum_sequential(v)
    assert np.float32(got).view(np.uint32) == np.float32(want).view(np.uint32), (got, want)
