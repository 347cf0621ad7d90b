"""Launches of at least 194,560 targets walk two neighbouring targets per lane, and
correction passes first take the removed particles out of their target list.  A
subhalo's results do not depend on the call it comes in, so a call of many
subhaloes (odd sizes: pairs that straddle two of them, an odd total) gives every
one of them the same bits as calls of a few, which stay below that line (the
small ones run all their passes in one launch, which has no such list)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(params, batch, cutoff=None):
    from hbtplus_gb300.unbind import Unbinder
    with Unbinder(params) as ub:
        if cutoff is not None:
            ub.set_option("small_cutoff", cutoff)
        return ub.unbind_batch(batch, check_status=False)


@pytest.mark.parametrize("sizes,theta", [
    ([1, 2, 3, 7, 1023, 1025, 1799] * 60, 0.45),
    ([33, 1801, 511] * 90, 0.7),
    ([97_281, 88_888], 0.45),
])
def test_large_launch_gives_each_subhalo_its_own_bits(sizes, theta):
    from hbtplus_gb300 import synthetic as S
    subs = [S.single_subhalo(n=n, seed=500 + i) for i, n in enumerate(sizes)]
    p = S.default_params(open_angle=theta)
    whole = S.concat(subs)
    off = whole["offsets"]
    assert off[-1] >= 194_560
    order, energy, res = run(p, whole, 0)
    step = max(1, len(subs) // 8)
    for a in range(0, len(subs), step):
        b = min(len(subs), a + step)
        part = S.concat(subs[a:b])
        o, e, r = run(p, part)
        lo = off[a]
        for j in range(b - a):
            n0, n1 = part["offsets"][j], part["offsets"][j + 1]
            assert np.array_equal(order[lo + n0:lo + n1], o[n0:n1])
            assert np.array_equal(energy[lo + n0:lo + n1].view(np.uint32), e[n0:n1].view(np.uint32))
            for k in r[j]:
                assert np.array_equal(np.asarray(res[a + j][k]), np.asarray(r[j][k])), k
