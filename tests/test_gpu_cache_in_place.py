"""nb_cache_infer with the outputs in the rows' own memory (n x 3 floats somewhere in the n x 64 read)
gives what it gives with a buffer of their own, bit for bit."""
import pytest
import torch

import nbounce_gb300 as nb
from nbounce_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [L.NB_CACHE_TCGEN05, L.NB_CACHE_MMA_SYNC])
@pytest.mark.parametrize("n", [1, 129, 100003])
def test_outputs_in_the_rows_memory(n, path):
    cache = nb.RadianceCache(seed=11, tensor_path=path)
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand(n, 64, generator=g, device="cuda")
    want = torch.empty(n, 3, device="cuda")
    cache.infer(x, n, want)
    for at in (0, 1, 61 * n // 2, 61 * n - 1, 61 * n):
        rows = x.clone()
        out = rows.view(-1)[at:at + 3 * n]
        cache.infer(rows, n, out)
        assert torch.equal(out.view(torch.int32), want.view(-1).view(torch.int32)), at
    # partly behind the rows' end and before their start
    for lead, at in ((0, 64 * n - n), (2 * n, 0)):
        flat = torch.empty(lead + 64 * n + 3 * n, device="cuda")
        rows = flat[lead:lead + 64 * n]
        rows.copy_(x.view(-1))
        out = flat[at:at + 3 * n]
        cache.infer(rows, n, out)
        assert torch.equal(out.view(torch.int32), want.view(-1).view(torch.int32)), (lead, at)
