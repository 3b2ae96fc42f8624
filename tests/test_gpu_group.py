"""FP64 products of blocks other than uniform 4 x 4 (the staged group kernel): block sizes at the edges of its
register tiles and of its 16-byte copies (odd and even, 1 to 16, one size and several), few and many output
blocks, operands on an odd 8-byte boundary, and the same products in a batch.  Reference rounding: the bits of
the oracle's default kernel."""
import numpy as np
import pytest

import blockmaps as bm
from cq_b200 import inputs
from cq_oracle import OracleSystem

pytestmark = pytest.mark.gpu

# name -> (cells per side, block size of atom k)
SIZES = {"u16": (2, lambda k: 16), "u9": (2, lambda k: 9), "u1": (2, lambda k: 1), "1to16": (2, lambda k: 1 + k % 16),
         "4_13_many": (3, lambda k: 13 if k % 3 == 0 else 4), "u13_many": (3, lambda k: 13)}


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("sizes", sorted(SIZES))
def test_group_kernel_bits(sizes, mult_type):
    import torch
    import cq_b200
    ncell, nd = SIZES[sizes]
    coords, cell = inputs.diamond_si(ncell, sigma=0.05, seed=41)
    nsf = np.array([nd(k) for k in range(len(coords))], np.int32)
    rc = [14.0, 6.0, 20.0] if mult_type == 2 else [6.0, 8.0, 14.0]
    o = OracleSystem(coords, cell, nsf, rc)
    g = cq_b200.System(coords, cell, nsf, rc)
    bls = [bm.oracle_blocklist(o, r, coords, cell) for r in range(3)]
    ops = [inputs.random_blocks(bls[r], 7 + r, inputs.TAG_RANDOM_A) for r in range(3)]
    out = 2 if mult_type == 1 else 0
    ref = [x.copy() for x in ops]
    ref[out][:] = 0.0
    o.mat_mult(mult_type, 0, 1, 2, *ref)
    if "many" in sizes:
        assert g.n_blocks(out) >= 148 * 18 * 4       # four output blocks per warp; the others run two
    for shift in (0, 1):                             # 16-byte aligned operands, then an odd multiple of 8 bytes
        dev = []
        for r in range(3):
            t = torch.full((len(ops[r]) + 1,), float("nan"), dtype=torch.float64, device="cuda")
            if r != out:
                t[shift:shift + len(ops[r])] = torch.from_numpy(ops[r])
            dev.append(t[shift:shift + len(ops[r])])
        torch.cuda.synchronize()
        g.mat_mult(mult_type, 0, 1, 2, *dev)
        g.synchronize()
        assert np.array_equal(dev[out].cpu().numpy(), ref[out])
        dev[out].fill_(float("nan"))
        torch.cuda.synchronize()
        cq_b200.mat_mult_batch([(g, mult_type, 0, 1, 2, *dev, cq_b200.PREC_FP64)])
        g.synchronize()
        assert np.array_equal(dev[out].cpu().numpy(), ref[out])
