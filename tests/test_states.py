"""The states of a call from arrays of their fields (unbind.state_array): one record per
subhalo of the offsets, equal to the record made row by row, from every form a
field may have; a field with too few rows or coordinates is refused, never
stretched over the subhaloes or left short of what the library reads."""
import ctypes as C

import numpy as np
import pytest
import torch

from hbtplus_gb300 import _lib, adjoint
from hbtplus_gb300.unbind import Unbinder, _state

FRAMES = ("ref_pos", "ref_vel", "mostbound_pos", "mostbound_vel")


def _batch(nsub=5, seed=1):
    rng = np.random.default_rng(seed)
    b = {k: rng.normal(0, 50, (nsub, 3)).astype(np.float32) for k in FRAMES}
    b["offsets"] = np.concatenate([[0], np.cumsum(rng.integers(0, 9, nsub))])
    b["mostbound_id"] = rng.integers(-1, 1 << 60, nsub)
    b["id"] = rng.integers(0, 1 << 60, int(b["offsets"][-1]))
    return b


def _by_row(b):
    return b"".join(bytes(_state(*(b[k][s] for k in FRAMES), b["mostbound_id"][s]))
                    for s in range(len(b["offsets"]) - 1))


@pytest.mark.parametrize("ids", [1, 4, 0])
def test_too_few_ids_are_refused(ids):
    b = _batch()
    b["mostbound_id"] = b["mostbound_id"][:ids]
    with pytest.raises(IndexError):
        Unbinder.make_states(b)


@pytest.mark.parametrize("field", FRAMES)
@pytest.mark.parametrize("shape", [(1, 3), (4, 3), (5, 1), (5, 2), (3,), (5,), (1,), (0, 3)])
@pytest.mark.parametrize("nsub", [5, 3])
def test_short_frames_are_refused(field, shape, nsub):
    b = _batch(nsub)
    if len(shape) == 2 and shape[0] >= nsub and shape[1] >= 3:
        return  # enough rows
    for form in (np.asarray, torch.from_numpy, np.ndarray.tolist):
        b[field] = form(np.ones(shape, np.float32))
        with pytest.raises((IndexError, TypeError)):
            Unbinder.make_states(b)


@pytest.mark.parametrize("shape", [(1, 3), (4, 3), (5, 1), (3,)])
def test_gradient_frames_are_refused(shape):
    whole, short = np.ones((5, 3), np.float32), np.ones(shape, np.float32)
    for frames in ((whole, short), (short, whole), (short, short)):
        with pytest.raises((IndexError, TypeError)):
            adjoint._states(5, *frames)
    with pytest.raises(IndexError):  # a frame for every offset
        adjoint._states(6, whole, whole)
    assert len(adjoint._states(4, whole, whole)) >= 4


def test_gradient_of_one_subhalo_takes_a_triple():
    x, v = np.arange(3, dtype=np.float32), np.arange(3, 6, dtype=np.float32)
    assert bytes(adjoint._states(1, x, v)) == bytes(adjoint._states(1, x[None], v[None]))
    for a, b in ((x[:2], v), (x, v[:1])):
        with pytest.raises((IndexError, TypeError)):
            adjoint._states(1, a, b)


FORMS = {
    "float64": lambda v: v.astype(np.float64) * (1 + 1e-9),
    "integers": lambda v: (v * 1e16).astype(np.int64),
    "lists": lambda v: v.tolist(),
    "tuple of arrays": lambda v: tuple(v),
    "tensor": lambda v: torch.from_numpy(v.copy()),
    "half tensor": lambda v: torch.from_numpy(v.copy()).to(torch.bfloat16),
    "list of tensors": lambda v: list(torch.from_numpy(v.copy())),
    "longer and wider": lambda v: np.pad(v, ((0, 3), (0, 2)), constant_values=7),
    "strided": lambda v: np.asfortranarray(np.repeat(v, 2, 0))[::2],
    "beyond float": lambda v: v.astype(np.float64) * 1e38,
    "objects": lambda v: v.astype(object),
}


@pytest.mark.parametrize("form", FORMS)
def test_states_are_the_rows(form):
    b = _batch()
    for k in FRAMES:
        b[k] = FORMS[form](b[k])
    want = _by_row(b)
    assert bytes(Unbinder.make_states(b)) == want
    dtype = np.uint64 if form == "integers" else np.int64
    column = torch.from_numpy(b["mostbound_id"].copy())[:, None]
    for ids in (b["mostbound_id"].tolist(), b["mostbound_id"].astype(dtype), column,
                np.append(b["mostbound_id"], 3)):
        assert bytes(Unbinder.make_states(dict(b, mostbound_id=ids))) == want


@pytest.mark.parametrize("nsub", [0, 1, 5])
def test_ids_default_to_each_lists_first(nsub):
    b = _batch(nsub, seed=3)
    off = b["offsets"]
    b["mostbound_id"] = [int(b["id"][off[s]]) if off[s + 1] > off[s] else -1 for s in range(nsub)]
    want = _by_row(b)
    del b["mostbound_id"]
    got = Unbinder.make_states(b)
    assert bytes(got)[:C.sizeof(_lib.hbtu_state) * nsub] == want


def test_only_the_lists_first_ids_are_copied(monkeypatch):
    from hbtplus_gb300 import unbind
    b = _batch(seed=4)
    del b["mostbound_id"]
    want = bytes(Unbinder.make_states(b))
    copied = []
    host = unbind._host
    monkeypatch.setattr(unbind, "_host", lambda v: copied.append(len(v)) or host(v))
    b["id"] = torch.from_numpy(b["id"].copy())
    assert bytes(Unbinder.make_states(b)) == want
    assert len(b["id"]) > 6 and max(copied) <= 6
    b["offsets"] = b["offsets"] + len(b["id"])
    with pytest.raises(IndexError):
        Unbinder.make_states(b)


@pytest.mark.parametrize("nsub", [1, 4, 5])
def test_few_and_many_states_are_the_same(nsub):
    b = _batch(nsub, seed=6)
    assert bytes(Unbinder.make_states(b)) == _by_row(b)
    tensors = {k: torch.from_numpy(v.copy()) if k in FRAMES else v for k, v in b.items()}
    assert bytes(Unbinder.make_states(tensors)) == _by_row(b)
