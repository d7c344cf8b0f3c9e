"""The Newton-Krylov path's K0 product and block-Jacobi blocks (csrc/pd_nk.cu) in every lane group, with
the eight warps that share a slice of a small body and the one warp of a large one (more than 3,552
slices: 4,200 points at 32 lanes a point), and slices of fewer rows than a warp takes at a time.
Reference and bars: the oracle's operators, 1e-5 (FP32) as in tests/test_gpu_nk.py."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import oracle_body
from jfnk import OracleNK
from pdcuda import newton_krylov as nkm
from test_gpu_nk import deformed_beam, rel
from test_nk_host import nk_conditions, small_beam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(7, 4, 2), (23, 7, 5), (30, 14, 10)])
@pytest.mark.parametrize("group", [1, 2, 8, 16, 32])
def test_operators(shape, group):
    body = small_beam(*shape)
    dev = pd.DeviceBody(body, precision="fp64")
    dev.set_mapping(group)
    ob = oracle_body(body)
    onk = OracleNK(ob, nk_conditions(body))
    nk = pd.NewtonKrylov(steps=1)
    nkm.setup(dev, nk)
    deformed_beam(dev, ob)
    v = np.random.default_rng(7).standard_normal(3 * dev.n)
    v[onk.cmask] = 0.0
    assert rel(nkm.apply_operator(dev, nk, "k0", v), onk.k0(v)) <= 1e-5
    nk.preconditioner = "block_jacobi"
    assert rel(nkm.apply_operator(dev, nk, "precond", v), onk.precond("block_jacobi", v)) <= 1e-6
    dev.close()
