"""The rule by which the leading axes of a product's input are counted as one axis of rows (`l3ci_row_stride`), against the
addresses of the rows themselves.  CPU only."""
import ctypes as C
import itertools

import pytest
import torch


def _by_addresses(sizes, strides):
    """The distance between consecutive rows in index order if it is one and the same and rows do not overlap, else -1."""
    if strides[-1] != 1 and sizes[-1] > 1:
        return -1
    starts = [sum(i * s for i, s in zip(at, strides)) for at in itertools.product(*(range(n) for n in sizes[:-1]))]
    steps = {b - a for a, b in zip(starts, starts[1:])}
    if not steps:
        return sizes[-1]
    return steps.pop() if len(steps) == 1 and min(b - a for a, b in zip(starts, starts[1:])) >= sizes[-1] else -1


@pytest.mark.parametrize("dims", [1, 2, 3, 4])
def test_every_order_of_sizes_and_strides(capi, dims):
    lib, n = capi.load(), 0
    for sizes in itertools.product(*([(1, 2, 3)] * (dims - 1)), (8, 16)):
        for strides in itertools.product(*([(0, 1, 8, 16, 24, 48)] * (dims - 1)), (1, 2)):
            got = lib.l3ci_row_stride((C.c_int64 * dims)(*sizes), (C.c_int64 * dims)(*strides), dims)
            assert got == _by_addresses(sizes, strides), (sizes, strides)
            n += got > 0
    assert n > 0


def test_broadcast_rows_are_not_rows_of_a_matrix(capi):
    base = torch.zeros(2, 64)
    for x in (base[:, None].expand(2, 3, 64), base[None].expand(3, 2, 64), base[:1].expand(5, 64), base[:, None, None].expand(2, 2, 3, 64)):
        assert capi._row_stride(x) is None
    for x, want in ((base, 64), (base[:, None], 64), (base[:1].expand(1, 64), 64), (torch.zeros(2, 3, 72)[..., :64], 72), (base[0], 64),
                    (torch.zeros(5, 3, 64)[:, -1], 192)):
        assert capi._row_stride(x) == want
    assert capi._row_stride(torch.zeros(5, 3, 64)[:, :2]) is None and capi._row_stride(base.t()) is None
