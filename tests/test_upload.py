"""Which arguments travel in the packed upload of small host arrays: nothing
that torch.as_tensor refuses, so such arguments are refused as without it, and
nothing in a graph capture."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("x", [
    np.array(["1.0"]), np.array([1.0, 2.0], dtype=object), np.arange(4.0)[::-1],
    np.arange(4, dtype=">f8"), np.arange(4, dtype=np.longdouble),
    np.array(["2020-01-01"], dtype="M8[D]")])
def test_refused_arrays_are_not_packed(x):
    from astroviper_b200 import _kernels as K
    with pytest.raises((TypeError, ValueError)):
        torch.as_tensor(x, dtype=torch.float64)
    assert not K._packable(x)


@pytest.mark.parametrize("x", [
    np.array([1, 2]), np.float64([1.5]), np.float32([[1.5, 2], [3, 4]]).T, np.arange(8)[::2],
    np.array([True]), np.zeros((3, 0)), np.array(3.0), np.arange(3, dtype=np.uint16)])
def test_packed_arrays_keep_values_and_shape(x):
    from astroviper_b200 import _kernels as K
    assert K._packable(x)
    a = np.ascontiguousarray(x, dtype=np.float64).reshape(x.shape)
    t = torch.as_tensor(x, dtype=torch.float64)
    assert tuple(t.shape) == a.shape and np.array_equal(t.numpy(), a)


@pytest.mark.gpu
def test_upload_matches_as_tensor():
    from astroviper_b200 import _kernels as K
    xs = [np.arange(5), [1.0, 2.0], torch.arange(3), np.array(3.0), np.zeros((2, 0)), (4, 5)]
    dts = [torch.int32, torch.float64, torch.int32, torch.float64, torch.float64, torch.int32]
    for got, x, dt in zip(K.upload(*zip(xs, dts)), xs, dts):
        want = torch.as_tensor(x, dtype=dt)
        assert got.is_cuda and got.dtype == dt and torch.equal(got.cpu(), want)
    with pytest.raises(TypeError):
        K.upload((np.array(["1.0"]), torch.float64))


@pytest.mark.gpu
def test_host_arrays_in_a_capture_are_refused():
    from astroviper_b200 import _kernels as K
    x = np.arange(5.0)
    K.upload((x, torch.float64))
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            K.upload((x, torch.float64))
    assert torch.equal(K.upload((x, torch.float64))[0].cpu(), torch.as_tensor(x))
