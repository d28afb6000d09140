"""The lattice test in front of the displacement kernels (no GPU needed)."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("cell,ok", [(np.eye(3) * 12.0, True), ([[11.0, 0, 0], [2, 9, 0], [-1.5, 3, 12]], True), (-np.eye(3), True),
                                     (np.diag([10.0, 10.0, 0.0]), False), ([[1.0, 2, 3], [4, 5, 6], [7, 8, 9]], False),
                                     ([[5.0, 0, 0], [5, 0, 0], [0, 0, 5]], False), (np.diag([10.0, 10.0, np.inf]), False),
                                     (np.diag([10.0, np.nan, 10.0]), False), (np.zeros((3, 3)), False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_regular_cells_pass(cell, ok, dtype):
    from so3lr_b200.api import _check_cell
    t = torch.as_tensor(np.asarray(cell), dtype=dtype)
    if ok:
        _check_cell(t)
    else:
        with pytest.raises(torch.linalg.LinAlgError):
            _check_cell(t)


@pytest.mark.parametrize("shape", [(9,), (2,), (1, 3, 3), (2, 3), (3, 2), (4, 4)])
def test_other_shapes_do_not(shape):
    from so3lr_b200.api import _check_cell
    with pytest.raises(ValueError):
        _check_cell(torch.ones(shape))


@pytest.mark.parametrize("edges,ok", [(12.0, True), ([12.0], True), ([12.0, 13.0, 14.0], True), ((9, 9, 9), True), (0.0, False), ([0.0], False),
                                      ([10.0, 10.0, 0.0], False), ([10.0, float("nan"), 10.0], False)])
@pytest.mark.parametrize("make", [lambda e: e, np.asarray, torch.as_tensor])
def test_boxes_given_by_their_edges(edges, ok, make):
    from so3lr_b200.api import _check_cell
    if ok:
        _check_cell(make(edges))
    else:
        with pytest.raises(torch.linalg.LinAlgError):
            _check_cell(make(edges))
