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


@pytest.mark.parametrize("sizes,sample", [
    ([1, 2, 3, 7, 1023, 1025, 1799] * 60, 64),
    ([33, 1801, 511] * 90, 300),
    ([64_007, 65, 80_001], 1000),
    ([200_003], 50),
])
def test_sampled_targets_in_either_order(sizes, sample):
    """With sampled potentials a large call sorts its targets along a space-filling
    curve and a small one takes them in list order: the same bits per subhalo.  (A
    large subhalo is checked beside one that shares its call: fewer than half of
    those particles are then targets in list order, and none is sorted.)"""
    from hbtplus_gb300 import synthetic as S
    subs = [S.single_subhalo(n=n, seed=900 + i) for i, n in enumerate(sizes)]
    p = S.default_params(max_sample_size=sample)
    whole = S.concat(subs)
    off = whole["offsets"]
    assert off[-1] >= 1 << 17
    order, energy, res = run(p, whole, 0)
    if len(sizes) == 1:  # N / 2 particles that are never targets: 1-particle subhaloes
        rest = S.concat([S.single_subhalo(n=1, seed=3) for _ in range(2)])
        n = int(off[-1]) + 1000
        pad = {k: np.concatenate([whole[k]] + [rest[k][:1]] * n) for k in ("pos", "vel", "mass", "id")}
        pad["offsets"] = np.concatenate([off, off[-1] + 1 + np.arange(n)])
        for k in whole:
            if k not in pad:
                pad[k] = np.concatenate([whole[k]] + [rest[k][:1]] * n)
        o, e, r = run(p, pad, 0)
        m = int(off[-1])
        assert np.array_equal(order, o[:m])
        assert np.array_equal(energy.view(np.uint32), e[:m].view(np.uint32))
        for k in res[0]:
            assert np.array_equal(np.asarray(res[0][k]), np.asarray(r[0][k])), k
        return
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
