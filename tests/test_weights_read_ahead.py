"""Kernels are launched while the ones before them still run.  A product may read its weight's first tiles before it waits for
those only if its caller says that none of them writes the weight."""
import inspect
import os
import re

import pytest
import torch

import rocml_b200
from rocml_b200 import kernels

CSRC = os.path.join(os.path.dirname(rocml_b200.__file__), "csrc")
DEV = "cuda:0"


@pytest.mark.parametrize("name", ["gemm_generic", "gemm_tcgen05", "gemm_tcgen05_act", "gemm_tcgen05_add", "gemm_tcgen05_qkv_rope"])
def test_a_weight_is_not_taken_for_complete_unless_the_caller_says_so(name):
    assert inspect.signature(getattr(kernels, name)).parameters["static_w"].default is False


@pytest.mark.parametrize("file,kernel,read", [
    ("gemm_generic.cu", "gemm_f32_cluster_kernel", "fetch_w(kt, kt)"), ("gemm_generic.cu", "gemm_rows_f32_kernel", "load_w(wv, k_lo)"),
    ("gemm_tcgen05.cu", "gemm_tcgen05_kernel", "tma_load_2d(sa, &map_a"), ("gemm_tcgen05.cu", "gemm_tcgen05_persistent_kernel", "&map_b, kb * BK"),
    ("gemm_tcgen05.cu", "gemm_tcgen05_pair_kernel", "&map_b, (j % n_kb)")])
def test_the_first_read_of_a_weight_follows_a_wait_that_only_that_word_lifts(file, kernel, read):
    with open(os.path.join(CSRC, file)) as f:
        body = f.read()
    body = body[re.search(r"\n%s\(" % kernel, body).end():]
    wait = re.search(r"if \(!(p\.)?w_ready\) (rb::)?pdl_wait\(\);", body)
    assert wait is not None and wait.end() < body.index(read)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [8, 40, 300])
def test_a_product_may_take_the_result_of_the_kernel_before_it_as_its_weight(M):
    """Cast, then multiply with what was cast, many times over with other values in the same buffer."""
    g = torch.Generator().manual_seed(1)
    for dtype, other in ((torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)):
        x = torch.randn((M, 512), generator=g).to(DEV).to(dtype)
        sources = [torch.randn((4096, 512), generator=g).to(DEV).to(other) for _ in range(4)]
        w = torch.zeros((4096, 512), dtype=dtype, device=DEV)
        outs = []
        torch.cuda.synchronize()
        for _ in range(3):
            for source in sources:
                out = torch.empty((M, 4096), dtype=torch.float32, device=DEV)
                kernels.cast(source, w)
                if dtype == torch.float32:
                    kernels.gemm_generic(x, w, out)
                else:
                    assert kernels.gemm_tcgen05(x, w, out)
                outs.append(out)
        for i, out in enumerate(outs):
            want = x.double() @ sources[i % 4].to(dtype).double().t()
            assert ((out.double() - want).abs().max() / want.abs().max()).item() < 1e-5
