"""CPU check of the bucket search of the selection (`csrc/dec_role.cuh`: `dec_prepare_floors`, `dec_select_chunk`): the first
bucket whose floor a magnitude reaches, found by halving over the running minimum of the floors, restated in Python with
the same steps and compared with the comparison of all floors.  The kernel itself is compared with the oracle on the GPU."""
import numpy as np
import pytest

from oracle import selection


def search(floors, mags):
    """running minimum that ignores NaN (fminf), then five halvings and a last comparison"""
    low = np.fmin.accumulate(floors.astype(np.float32))
    pos = np.zeros(mags.shape, int)
    with np.errstate(invalid="ignore"):
        for d in (16, 8, 4, 2, 1):
            pos += np.where(~(mags >= low[pos + d - 1]), d, 0)
        return np.where(np.isfinite(mags) & (mags >= low[pos]), pos, 32)


def all_floors(floors, mags):
    with np.errstate(invalid="ignore"):
        reached = mags[:, None] >= floors[None, :].astype(np.float32)
    return np.where(reached.any(1) & np.isfinite(mags), reached.argmax(1), 32)


@pytest.mark.parametrize("dtype", ["fp16", "bf16", "fp32"])
@pytest.mark.parametrize("a,b", [(60.0, 2.5), (3.0, 3.0), (5000.0, 0.25), (0.0, 0.0), (1.0, -1.0), (np.inf, 1.0), (np.nan, 1.0), (2.0, np.nan)])
def test_search_finds_the_first_floor(dtype, a, b):
    with np.errstate(all="ignore"):
        floors = selection.bucket_floors(a, b, dtype)
    rng = np.random.default_rng(3)
    mags = np.abs(rng.standard_normal(2000)).astype(np.float32) * 3
    finite = floors[np.isfinite(floors)].astype(np.float32)
    mags = np.concatenate([mags, finite, np.nextafter(finite, np.float32(np.inf)), np.nextafter(finite, np.float32(-np.inf)),
                           np.array([0.0, np.inf, np.nan, 65504.0], np.float32)])
    mags = np.abs(mags)
    assert np.array_equal(search(floors, mags), all_floors(floors, mags))


@pytest.mark.parametrize("seed", range(20))
def test_search_with_floors_in_any_order(seed):
    rng = np.random.default_rng(seed)
    floors = np.abs(rng.standard_normal(32)).astype(np.float32)
    floors[rng.integers(0, 32, 3)] = np.nan
    floors[rng.integers(0, 32, 2)] = np.inf
    if seed % 2:
        floors[0] = np.nan
    mags = np.abs(rng.standard_normal(500)).astype(np.float32)
    assert np.array_equal(search(floors, mags), all_floors(floors, mags))
