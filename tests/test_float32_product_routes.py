"""Which kernel takes a float32 product: at sizes where one of the two was measured at least a tenth quicker, and where the
tensor cores' error would be the larger one.  No GPU."""

import pytest
import torch

from tinyvllm_b200.ops import kernels
from tinyvllm_b200.ops.linear import linear

TENSOR = [(33, 4096, 4096), (48, 4096, 1024), (64, 6144, 1024), (301, 1024, 3072), (677, 1024, 2048), (2048, 6144, 1024),
          (301, 64, 512), (2048, 64, 256), (192, 64, 128), (677, 256, 2048), (8192, 128, 1024), (2048, 4096, 64), (8192, 2048, 48)]
CORES = [(32, 4096, 4096), (9, 1024, 3072), (33, 64, 64), (301, 512, 64), (2048, 128, 64), (8192, 128, 64), (2048, 256, 128),
         (301, 64, 32), (8192, 512, 32), (2048, 64, 2048), (8192, 8, 2048), (8192, 64, 4096), (1024, 8, 4096), (8192, 64, 8192),
         (2048, 12288, 12), (64, 64, 4), (677, 1024, 8)]


class OnGpu(torch.Tensor):
    is_cuda = True


@pytest.mark.parametrize("sizes,kernel", [(s, "gemm_f32_tc") for s in TENSOR] + [(s, "gemm_nt_simt") for s in CORES])
def test_route(monkeypatch, sizes, kernel):
    taken = []
    for name in ("gemm_f32_tc", "gemm_nt_simt"):
        monkeypatch.setattr(kernels, name, lambda *args, name=name, **words: taken.append(name))
    m, n, k = sizes
    linear(torch.empty(m, k).as_subclass(OnGpu), torch.empty(n, k))
    assert taken == [kernel]
    # rows off the 16-byte boundary are the float32 cores' in any case
    linear(torch.empty(m * k + 1)[1:].view(m, k).as_subclass(OnGpu), torch.empty(n, k))
    assert taken[1] == "gemm_nt_simt"


@pytest.mark.parametrize("shape,dtype,kernel", [((64, 6144), torch.float32, "gemm_f32_tc"), ((70, 6144), torch.float32, "gemm_nt_simt"),
                                                ((64, 6150), torch.float32, "gemm_nt_simt"), ((64, 6144), torch.bfloat16, "gemm_nt_simt")])
def test_a_result_inside_a_larger_tensor_or_of_another_type(monkeypatch, shape, dtype, kernel):
    """The float32 cores' kernels write the first rows and columns of whatever they are given."""
    taken = []
    for name in ("gemm_f32_tc", "gemm_nt_simt"):
        monkeypatch.setattr(kernels, name, lambda *args, name=name, **words: taken.append(name))
    linear(torch.empty(64, 1024).as_subclass(OnGpu), torch.empty(6144, 1024), out=torch.empty(shape, dtype=dtype))
    assert taken == [kernel]


def test_operands_that_are_not_matrices_are_refused_as_ever(monkeypatch):
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    for x in (torch.tensor(1.0), torch.empty(1024), torch.empty(2, 40, 1024)):
        with pytest.raises(kernels.KernelError):
            linear(x.as_subclass(OnGpu), torch.empty(6144, 1024))
