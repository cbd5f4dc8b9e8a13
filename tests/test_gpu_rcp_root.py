"""phys::rcp and phys::root (device/physics.cuh) against 1/x and sqrt.

Bound: the iterations leave a relative error far below 2^-60 before the last fused operation, which rounds once,
so the results are within half an ulp and a little of the exact ones and within one ulp of the correctly
rounded ones.  Outside normal numbers they do what their comments say."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

from dg_b200 import build

pytestmark = pytest.mark.gpu
INF, NAN, TINY = np.inf, np.nan, 5e-324


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    so = tmp_path_factory.mktemp("cuda") / "librcp_root.so"
    src = Path(__file__).parent / "cuda" / "rcp_root.cu"
    subprocess.run([build.NVCC, *build.NVFLAGS, f"-I{build.SRC}", "-shared", str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))

    def run(what, x):
        xd = torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda()
        yd = torch.empty_like(xd)
        assert lib.rcp_root(what, xd.numel(), C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr())) == 0
        return yd.cpu().numpy()

    return run


@pytest.mark.parametrize("span", [40, 500])  # magnitudes 1e-12 .. 1e12, and 1e-150 .. 1e150
def test_within_one_ulp(apply, span):
    rng = np.random.default_rng(span)
    x = np.ldexp(1 + rng.random(1 << 22), rng.integers(-span, span, 1 << 22))
    x[:8] = [1, 2, 4, 0.5, 1 + 2.0 ** -52, 2 - 2.0 ** -52, 3, 1 / 3]
    for what, y, want in ((0, apply(0, x), 1 / x), (0, apply(0, -x), -1 / x), (1, apply(1, x), np.sqrt(x))):
        assert (np.abs(y - want) <= np.spacing(np.abs(want))).all()
    assert (np.mean(apply(0, x) != 1 / x) < 1e-5) and (np.mean(apply(1, x) != np.sqrt(x)) < 1e-5)


def test_edges(apply):
    x = np.array([0.0, -0.0, TINY, -TINY, 2.0 ** -1022, INF, -INF, NAN, -4.0, 2.0 ** 1022])
    want_rcp = [NAN, NAN, NAN, NAN, 2.0 ** 1022, NAN, NAN, NAN, -0.25, 0.0]
    want_root = [0.0, 0.0, 0.0, 0.0, 2.0 ** -511, NAN, NAN, NAN, NAN, 2.0 ** 511]
    rcp, root = apply(0, x), apply(1, x)
    keep = np.arange(len(x)) != 9  # 1/2^1022 is the smallest normal number: 0 or itself
    assert np.array_equal(rcp[keep], np.array(want_rcp)[keep], equal_nan=True) and rcp[9] in (0.0, 2.0 ** -1022)
    assert np.array_equal(root, want_root, equal_nan=True)
