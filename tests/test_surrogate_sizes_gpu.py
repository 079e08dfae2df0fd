"""Surrogate kernels at the sizes where they can go wrong: the feature rows
around the register sort's widths, and the GEMM with more tiles than SMs (four
stages) for fewer, as many and more K steps than stages."""
import ctypes

import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required")
    return torch


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257])
def test_feature_rows(torch, n):
    from brkga_fft2_b200.evaluator import _NativeProblem
    from brkga_fft2_b200.surrogate import Surrogate
    inst = instances.make_instance("f", n, [(40, 40), (50, 36), (44, 44)], 2, bbox_min=3, bbox_max=20,
                                   scale_machines=True)
    pk = pack_problem(inst.problem_data, n, inst.nb_machines, inst.thresholds, inst.instance_parts)
    native = _NativeProblem(pk)
    ch = instances.chromosomes(19, n, 8)
    ch[0, : n // 2] = ch[0, n - 1]
    ch[1, n:] = 0.9  # every part on one machine
    for kind, ref in (("decode", mo.features), ("order", mo.order_features)):
        sur = Surrogate(native, max_batch=128, buffer_capacity=200, seed=3, features=kind)
        np.testing.assert_array_equal(sur.features(torch.from_numpy(ch).cuda()), ref(pk, ch, sur.in_pad))
        sur.close()


@pytest.mark.parametrize("M,N,K", [(128 * 75, 128, 64), (128 * 75, 128, 256), (128 * 75, 128, 320), (128 * 38, 256, 640),
                                   (128 * 149, 64, 512)])
def test_gemm_of_more_tiles_than_sms(torch, M, N, K):
    lib = abi.load_library()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    C = torch.full((M, N), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = lib.brkga_gemm_bf16(ctypes.c_void_p(A.data_ptr()), K, ctypes.c_void_p(B.data_ptr()), K,
                             ctypes.c_void_p(C.data_ptr()), N, M, N, K, ctypes.c_void_p(err.data_ptr()),
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    # fp32 matmul of the same bf16 operands: products are exact, K-term sums differ by rounding only
    torch.testing.assert_close(C, A.float() @ B.float().T, rtol=1e-4, atol=1e-3)
