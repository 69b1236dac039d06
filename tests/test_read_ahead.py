"""Kernels are launched while the ones before them still run.  A product may read its weight's first tiles, and decode attention
the rows of the new token's page, before it waits for those only if its caller says that none of them writes there."""
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


def test_rows_beside_the_new_one_are_not_taken_for_complete_unless_the_caller_says_so():
    assert inspect.signature(kernels.attention_decode_fused).parameters["static_rows"].default is False
    with open(os.path.join(CSRC, "attention_decode.cu")) as f:
        text = f.read()
    assert "const bool patch = owner && pj.rows_ready &&" in text         # the page is copied early only where the new row is patched in
    early = re.search(r"const bool early0 = ([^;]*);", text).group(1)
    assert early == "page_first < new_page || (patch && page_first == new_page)"


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 40, 64, 100])
def test_decode_attention_may_follow_the_kernel_that_writes_the_rows_before_the_new_one(n):
    """A prompt's rows cached by one kernel and a token decoded by the next: the same bits as with a wait between them."""
    hd, nq, nkv = 128, 8, 2
    width, T = (nq + 2 * nkv) * hd, n - 1
    g = torch.Generator().manual_seed(n)
    table = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV)
    one = lambda v: torch.tensor([v], dtype=torch.int32, device=DEV)  # noqa: E731
    pos, slots = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    cu, kv, slot = torch.tensor([0, 1], dtype=torch.int32, device=DEV), one(n), one(0)
    got = {False: [], True: []}
    prompts = [torch.randn((T, width), generator=g).to(DEV).bfloat16() for _ in range(6)]
    token = torch.randn((2, 1, width), generator=g).to(DEV)
    k, v = (torch.zeros((2, nkv, 64, hd), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    q = torch.empty((T, nq * hd), dtype=torch.bfloat16, device=DEV)
    acc, ml = torch.empty((1, nq, 2, hd), device=DEV), torch.empty((1, nq, 2, 2), device=DEV)
    outs = [torch.empty((1, nq * hd), dtype=torch.bfloat16, device=DEV) for _ in range(12)]
    torch.cuda.synchronize()
    for wait in (True, False):
        for p in prompts:
            out = outs.pop()
            kernels.qk_norm_rope_cache(p, q, T, nq, nkv, hd, None, None, 1e-6, None, 0, pos, slots, table, k, v)
            if wait:
                torch.cuda.synchronize()
            assert kernels.attention_decode_fused(token, out, k, v, table, slot, cu, kv, 1, nq, nkv, hd, None, None, 1e-6, None, True,
                                                  0.1, 0, 1, acc, ml, 2)
            got[wait].append(out)
    for a, b in zip(got[True], got[False]):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
