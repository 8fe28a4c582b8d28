"""DeviceAtoms from each kind of array: values and shapes, and no ties between the
three device arrays."""
import numpy as np
import pytest
import torch

from problems import make_atoms

pytestmark = pytest.mark.gpu


class DeviceArray:
    """An array of another library in device memory."""

    def __init__(self, t):
        self._t = t
        self.shape, self.ndim = tuple(t.shape), t.dim()

    @property
    def __cuda_array_interface__(self):
        return self._t.__cuda_array_interface__

    def __array__(self, *a, **k):
        raise TypeError("implicit conversion to a host array is not allowed")


CAST = {"numpy": np.asarray, "float64 cpu tensor": torch.from_numpy, "list": lambda a: a.tolist(),
        "list of tensors": lambda a: list(torch.from_numpy(a).reshape(-1).cuda())
        if a.ndim == 1 else a,
        "cuda tensor": lambda a: torch.from_numpy(a).cuda(),
        "device array": lambda a: DeviceArray(torch.from_numpy(a).cuda()),
        "device array and host": lambda a: a if a.ndim == 1
        else DeviceArray(torch.from_numpy(a).float().cuda())}


@pytest.mark.parametrize("kind", CAST)
@pytest.mark.parametrize("dim,iso", [(2, False), (3, True)])
def test_arrays_of_every_kind(eng, cuda_ready, kind, dim, iso):
    I, x, r = make_atoms(dim, 5, dim, iso=iso)
    at = eng.DeviceAtoms(*(CAST[kind](a) for a in (I, x, r)))
    assert at.n == 5 and at.dim == dim and at.iso == iso
    assert torch.equal(at.I.cpu(), torch.from_numpy(I).float())
    assert torch.equal(at.x.cpu(), torch.from_numpy(x).float())
    assert torch.equal(at.r.cpu(), torch.from_numpy(r[:, 0] if iso else r).float())


@pytest.mark.parametrize("iso", [False, True])
def test_one_arrays_change_is_its_own(eng, cuda_ready, iso):
    """An array saved for a backward pass stays valid when another one changes."""
    I, x, r = make_atoms(3, 5, 1, iso=iso)
    at = eng.DeviceAtoms(I, x, r)
    y = (at.I.requires_grad_() ** 2).sum()
    with torch.no_grad():
        at.x += 1.0
        at.r *= 2.0
    y.backward()
    assert torch.equal(at.I.grad, 2 * at.I.detach())
    assert torch.allclose(at.x.cpu(), torch.from_numpy(x).float() + 1)
