"""The caller's encoded rows as nb_cache_infer / _gradient read them: every row of a batch gives the
same bits whatever the batch size (full and ragged groups of 128 rows, one and several rounds of the
grid) and whatever the alignment of the caller's buffers."""
import numpy as np
import pytest
import torch

import nbounce_gb300 as nb

pytestmark = pytest.mark.gpu

N = 200003  # the largest batch: several rounds of 512 rows per block


def _at(values, offset):
    """A device copy that starts `offset` floats into its buffer (offset 1: 4-byte aligned only)."""
    flat = torch.empty(values.numel() + offset, device="cuda")
    flat[offset:] = values.reshape(-1)
    return flat[offset:]


@pytest.fixture(scope="module")
def rows():
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand(N, 64, generator=g, device="cuda") * 2.0 - 0.5
    x[:, 62] = 1.0
    x[3, 5] = float("nan")
    x[4, 6] = float("inf")
    x[130] = 0.0
    y = torch.rand(N, 3, generator=g, device="cuda")
    cache = nb.RadianceCache(seed=11)
    whole = torch.empty(N, 3, device="cuda")
    cache.infer(x, N, whole)
    return cache, x, y, whole


@pytest.mark.parametrize("offset", [0, 1, 3, 4])
@pytest.mark.parametrize("n", [1, 7, 8, 31, 33, 127, 128, 129, 511, 513, 4097, N])
def test_rows_do_not_depend_on_batch_or_alignment(rows, n, offset):
    cache, x, _, whole = rows
    out = torch.full((n + 2, 3), 7.0, device="cuda")
    cache.infer(_at(x[:n], offset), n, out)
    assert torch.equal(out[:n].view(torch.int32), whole[:n].view(torch.int32))
    assert bool((out[n:] == 7.0).all())


@pytest.mark.parametrize("n", [1, 9, 127, 128, 129, 1000])
def test_gradient_does_not_depend_on_alignment(rows, n):
    cache, x, y, _ = rows
    got = []
    for offset in (0, 1):
        grad = torch.zeros(nb.cache.N_PARAMS, device="cuda")
        loss = cache.gradient(_at(x[200:200 + n], offset), _at(y[200:200 + n], offset), n, grad)
        got.append((loss, grad.cpu().numpy()))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1]) and np.abs(got[0][1]).max() > 0


@pytest.mark.parametrize("n", [128, 128 * 15 + 5, 128 * 64, 128 * 129 + 1])
def test_gradient_sums_all_groups(rows, n):
    """The mean gradient of a batch against the row-weighted mean of its parts' (FP32 sums of up to 130
    partials: relative 2-norm error below 1e-5), the loss likewise."""
    cache, x, y, _ = rows
    x, y = x[1000:1000 + n], y[1000:1000 + n]
    whole = torch.zeros(nb.cache.N_PARAMS, device="cuda")
    loss = cache.gradient(x, y, n, whole)
    total, losses = np.zeros(nb.cache.N_PARAMS), 0.0
    for k in range(0, n, 128):
        m = min(128, n - k)
        part = torch.zeros(nb.cache.N_PARAMS, device="cuda")
        losses += cache.gradient(x[k:].contiguous(), y[k:].contiguous(), m, part) * m
        total += part.cpu().numpy().astype(np.float64) * m
    err = np.linalg.norm(whole.cpu().numpy() - total / n) / np.linalg.norm(total / n)
    assert err < 1e-5 and abs(loss - losses / n) < 1e-5 * abs(loss)
