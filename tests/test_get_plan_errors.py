"""``get_plan`` refuses constants with the plan's own errors, whatever they are."""
import numpy as np
import pytest
import torch

from licom4py_gpu_b200.barotr import get_plan

BAD = {
    "lists": ([[0.0]] * 17, TypeError, "expected a torch.Tensor or numpy.ndarray, got list"),
    "none": ([None] * 17, TypeError, "got NoneType"),
    "too few": ([np.zeros((6, 14, 14))] * 2, ValueError, "17 CONST_SOURCES"),
    "shape": ([np.zeros((5, 14, 14))] * 17, ValueError, "has shape"),
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="the error without a GPU")
@pytest.mark.parametrize("name", BAD)
def test_without_a_gpu(name):
    with pytest.raises(RuntimeError, match="needs a CUDA device"):
        get_plan(BAD[name][0], device="cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("name", BAD)
def test_bad_constants(name):
    consts, error, text = BAD[name]
    with pytest.raises(error, match=text):
        get_plan(consts)
