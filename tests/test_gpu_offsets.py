"""Offsets that fall: rows that are valid one by one can then be more, and longer in
sum, than the neighbour array, so the build's list of long rows (over 4,096 entries)
must not grow past what rising offsets could make of it.  Such a build is refused
and the next one is sound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (selection, layout): the prefix build and the general one.
ROUTES = [("lower", "hybrid"), ("all", "uint"), ("lower", "bs"), ("lower", "pshort"), ("mask", "hybrid")]


@pytest.mark.parametrize("selection,layout", ROUTES)
@pytest.mark.parametrize("length", [4097, 5000])
def test_more_long_rows_than_the_neighbour_array_holds(eh, selection, layout, length):
    import torch
    n = 6001  # every second row is [0, length); the list has room for two
    off = np.zeros(n + 1, np.uint64)
    off[1::2] = length
    nbr = np.arange(length, dtype=np.uint32)
    mask = np.ones(length, np.uint8) if selection == "mask" else None
    with pytest.raises(eh.EHError) as ei:
        eh.Matrix.build(off, nbr, selection=selection, layout=layout, mask=mask)
    assert ei.value.status == 1 and "offsets" in str(ei.value)
    d_off = torch.from_numpy(off.view(np.int64)).cuda()
    d_nbr = torch.from_numpy(nbr.view(np.int32)).cuda()
    d_mask = None if mask is None else torch.from_numpy(mask).cuda()
    with pytest.raises(eh.EHError) as ei:
        eh.Matrix.build_device(n, d_off.data_ptr(), d_nbr.data_ptr(), selection=selection, layout=layout,
                               d_mask=None if d_mask is None else d_mask.data_ptr())
    assert ei.value.status == 1 and "offsets" in str(ei.value)
    # One such row with rising offsets is measured as ever.
    good = np.full(n + 1, length, np.uint64)
    good[:n] = 0
    m = eh.Matrix.build(good, nbr, selection=selection, layout=layout, mask=mask)
    assert m.info()["cardinality"] == length
