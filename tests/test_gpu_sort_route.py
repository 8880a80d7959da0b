"""Which way a sort goes: one CTA up to 3968 rows, the sample sort for keys that
rarely repeat, the radix passes for few values, for keys that repeat often, for few
varying bytes and for a memory budget without room for the buckets."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops
from tests.test_gpu_sort_spill import kernels, launched

pytestmark = pytest.mark.gpu
N = 1_000_003


def column(kind, r):
    if kind == "one leaf":
        return r.random(3968)
    if kind == "one level":
        return r.random(300_001)
    if kind == "uniform":
        return r.random(N)
    if kind == "wide ints":
        return r.integers(-2**62, 2**62, N)
    if kind == "few values":
        return r.integers(0, 12, N)
    if kind == "many of each":
        return r.integers(0, N // 40, N) * 0x1234567890AB
    if kind == "a tenth of one value":
        return np.where(r.random(N) < 0.1, 0.5, r.random(N))
    assert kind == "three bytes"
    return r.integers(0, 1 << 24, N)


ROUTES = {"one leaf": "big_leaf", "one level": "leaf", "uniform": "leaf", "wide ints": "leaf", "few values": "radix",
          "many of each": "radix", "a tenth of one value": "radix", "three bytes": "radix"}


def route(names):
    if launched(names, "radix_scatter_kernel"):
        return "radix"
    return "leaf" if launched(names, "msd_leaf_kernel") else "big_leaf"


@pytest.mark.parametrize("kind", list(ROUTES))
def test_route(db, kind):
    v = column(kind, np.random.default_rng(len(kind)))
    d = torch.from_numpy(v).cuda()
    got = []
    names = kernels(lambda: got.append(ops.sort(db, d, len(v), False)))
    assert route(names) == ROUTES[kind]
    assert np.array_equal(got[0][:len(v)].cpu().numpy(), np.argsort(v, kind="stable"))


def test_a_small_budget():
    v = np.random.default_rng(1).random(2_000_000)
    d = torch.from_numpy(v).cuda()
    with F.Database(0, mem_budget=256 << 20) as small:  # the buckets: 120 MB, above a quarter of it
        got = []
        assert route(kernels(lambda: got.append(ops.sort(small, d, len(v), True)))) == "radix"
        assert np.array_equal(got[0][:len(v)].cpu().numpy(), np.argsort(-v, kind="stable"))
