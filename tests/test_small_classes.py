"""The size classes of the per-subhalo kernel (small.cu): one warp, four warps or
a block or cluster per subhalo, by list length and by how many lists there are.
Whatever the class, a call's outputs must equal the batch path's (small_cutoff
0) bit for bit: at the edges of the classes, alone and among many, with sampled
potentials and their refinement, and with several particle types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(sizes, seed, types=False):
    from hbtplus_gb300 import synthetic as S
    rng = np.random.Generator(np.random.PCG64(seed))
    subs = []
    for n in sizes:
        k = max(n - n // 6, 0)
        subs.append(S.nfw_subhalo(rng, k, 0.2 * (max(n, 1) / 1e5) ** (1 / 3), 10.0,
                                  contaminant_frac=(n - k) / k if k else 0.0,
                                  center=rng.uniform(0, 100, 3)))
    S._assign_ids(rng, subs)
    b = S.concat(subs)
    assert np.array_equal(np.diff(b["offsets"]), sizes)
    if types:
        b["type"] = rng.integers(0, 7, len(b["mass"])).astype(np.int32)  # 6: not counted
        b["id"][rng.integers(0, len(b["id"]), 40)] = -1
    return b


def _same(b, **over):
    from hbtplus_gb300 import synthetic as S
    from hbtplus_gb300.unbind import Unbinder
    out = []
    for cutoff in (0, 2048):
        with Unbinder(S.default_params(**over), precision=0) as ub:
            ub.set_option("small_cutoff", cutoff)
            out.append(ub.unbind_batch(b))
            assert (ub.stats()["passes"] == 0) == (cutoff > 0)
    (oa, ea, ra), (ob, eb, rb) = out
    assert np.array_equal(oa, ob) and np.array_equal(ea, eb, equal_nan=True)
    for s, (x, y) in enumerate(zip(ra, rb)):
        assert all(np.array_equal(x[k], y[k]) for k in x), (s, x, y)
    return oa, ra


@pytest.mark.parametrize("n", [2, 31, 33, 64, 65, 128, 129, 512, 513, 1024, 1025, 2047, 2048])
def test_one_list(n):
    _same(_batch([n], n))


@pytest.mark.parametrize("sizes,over", [
    ([2048, 1025, 1024, 600, 513, 512, 511, 257, 256] + [130, 129, 128, 127, 65, 33, 20, 1, 0] * 6, {}),
    ([700] * 3 + [200] * 30 + [60] * 40, dict(max_sample_size=100)),
    ([300] * 5 + [129, 128] * 10 + [40] * 1300, {}),      # short lists: two warps each
    ([140] * 700 + [21] * 2500, dict(periodic=0)),        # medium: four warps; short: one warp
])
def test_many_lists(sizes, over):
    _same(_batch(sizes, len(sizes)), **over)


def test_particle_types():
    b = _batch([1500, 400, 90, 60, 40], 3, types=True)
    order, res = _same(b)
    for s, r in enumerate(res):
        if r["nbound"] <= 1:
            continue
        rows = int(b["offsets"][s]) + order[b["offsets"][s]:b["offsets"][s] + r["nbound"]]
        t = b["type"][rows]
        if r["nbound"] <= 100:
            t = np.where(b["id"][rows] == -1, 6, t)
        assert r["nbound_type"].tolist() == [int((t == q).sum()) for q in range(6)]
        m = [b["mass"][rows][t == q].astype(np.float64).sum() for q in range(6)]
        assert np.allclose(r["mbound_type"], m, rtol=2e-7, atol=0)
