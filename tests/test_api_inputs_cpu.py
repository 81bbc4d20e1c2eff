"""How the Python layer takes its inputs, as far as that needs no GPU."""
import numpy as np
import pytest
import torch

from skywalker_b200.api import Context, SkwError, _host_u32


@pytest.mark.parametrize("x", [
    np.arange(5, dtype=np.uint32), np.arange(-2, 3, dtype=np.int32), np.arange(5), [1, 2, 3], range(4), np.uint32(7), 7,
    np.array(7, np.uint32), np.array(7, np.int32), np.arange(10, dtype=np.uint32)[::2], np.arange(6, dtype=np.uint32).reshape(2, 3),
    np.arange(5, dtype=">u4"), np.ma.masked_array(np.arange(4, dtype=np.uint32)), np.zeros(0, np.uint32),
    np.frombuffer(b"\x00" + bytes(range(16)), np.uint8)[1:17].view("u4"),
    torch.arange(5, dtype=torch.int32), torch.tensor(7, dtype=torch.int32), torch.arange(6), torch.arange(9, dtype=torch.int32)[::2],
    torch.zeros(0, dtype=torch.int32)], ids=repr)
def test_start_vertices_are_taken_as_a_conversion_takes_them(x):
    want = np.ascontiguousarray(x, np.uint32)
    got = _host_u32(x)
    assert len(got) == len(want)
    data = got.numpy() if isinstance(got, torch.Tensor) else np.asarray(got)
    assert data.shape == want.shape and data.flags.c_contiguous and data.dtype.itemsize == 4 and data.dtype.isnative
    assert np.array_equal(data.view(np.uint32), want)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("make", [lambda: torch.zeros(4, dtype=torch.complex32),
                                  lambda: torch.zeros(4, dtype=torch.int32, device="meta"),
                                  lambda: torch.quantize_per_tensor(torch.ones(4), 0.1, 0, torch.qint32),
                                  lambda: torch.zeros(4, dtype=torch.int32).to_sparse()], ids=["complex32", "meta", "qint32", "sparse"])
def test_what_a_conversion_refuses_is_refused(make):
    with pytest.raises(Exception):
        np.ascontiguousarray(make(), np.uint32)
    with pytest.raises(Exception):
        _host_u32(make())


def test_no_conversion_where_none_is_needed():
    for x in (np.arange(5, dtype=np.uint32), np.arange(5, dtype=np.int32), torch.arange(5, dtype=torch.int32)):
        assert _host_u32(x) is x


class _Count:
    """A fan-out that is a number to ctypes, equal to none, and may change."""

    def __init__(self, n):
        self.n = n

    def __index__(self):
        return self.n


def test_khop_layout_goes_by_the_numbers():
    changing = [_Count(25), _Count(10)]
    assert Context.khop_layout(changing) == (276, 26)
    changing[0].n = 2
    assert Context.khop_layout(changing) == (23, 3)
    assert Context.khop_layout(np.array([25, 10])) == Context.khop_layout(torch.tensor([25, 10])) == (276, 26)
    for refused in ([25.0, 10], [], [1] * 5, [0, 3], [1 << 16, 1 << 16]):
        for _ in range(2):                 # after the same numbers were accepted, and after a refusal
            with pytest.raises((TypeError, SkwError)):
                Context.khop_layout(refused)
