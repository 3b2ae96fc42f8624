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


@pytest.mark.parametrize("shape", ["cell", "cluster33", "cluster1"])
@pytest.mark.parametrize("exact", [True, False])
def test_4x4_kernels_give_the_same_bits(shape, exact):
    """The staged 4 x 4 kernels against the unstaged one (one lane per element, checked against the oracle elsewhere):
    full and ragged groups of output blocks, pair lists that hold a whole row of B and lists that hold part of it
    (the input range shorter than the sum of the others), both mult types."""
    import torch
    import cq_b200
    coords, cell = {"cell": lambda: inputs.diamond_si(2, sigma=0.1, seed=51),
                    "cluster33": lambda: inputs.si_cluster(33, sigma=0.1, seed=52),
                    "cluster1": lambda: inputs.si_cluster(1, sigma=0.0, seed=53)}[shape]()
    g = cq_b200.System(coords, cell, np.full(len(coords), 4, np.int32), [10.0, 8.0, 18.0, 14.0])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    for t, rc in ((1, 2), (1, 3), (2, 2), (2, 3)):
        ops = [torch.rand(g.length(r), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for r in (0, 1, rc)]
        out = 2 if t == 1 else 0
        ref = None
        for v in (0, 3, 4, 5, -1):
            g.set_mult_variant(v)
            ops[out].fill_(float("nan"))
            torch.cuda.synchronize()
            g.mat_mult(t, 0, 1, rc, *ops, exact=exact)
            g.synchronize()
            ref = ops[out].clone() if ref is None else ref
            assert torch.equal(ops[out], ref), (t, rc, v)


@pytest.mark.parametrize("nd", ["4", "13", "4_13"])
def test_transpose_and_sums_against_index_arithmetic(nd):
    """Transposes and sums of equal and different ranges, element by element: 4 x 4 blocks (aligned, then on an odd
    8-byte boundary), 13 x 13 and both; a sum with itself keeps the two steps of the reference (scale, then add)."""
    import torch
    import cq_b200
    coords, cell = inputs.si_cluster(37, sigma=0.1, seed=61)
    nsf = np.array([{"4": 4, "13": 13, "4_13": 13 if k % 3 == 0 else 4}[nd] for k in range(len(coords))], np.int32)
    g = cq_b200.System(coords, cell, nsf, [9.0, 13.0])
    bls = [g.blocklist(r, coords, cell) for r in range(2)]
    vals = [inputs.random_blocks(bls[r], 3 + r, inputs.TAG_RANDOM_A) for r in range(2)]
    short, wide = bm.block_dict(bls[0]), bm.block_dict(bls[1])
    for shift in (0, 1):
        dev = []
        for v in vals + [np.zeros(bls[0].length)]:
            t = torch.zeros(len(v) + 1, dtype=torch.float64, device="cuda")
            t[shift:shift + len(v)] = torch.from_numpy(v)
            dev.append(t[shift:shift + len(v)])
        a, b, at = dev
        torch.cuda.synchronize()
        g.transpose(0, a, at)
        g.synchronize()
        assert np.array_equal(at.cpu().numpy(), bm.kat_transpose(bls[0], vals[0]))
        g.matrix_sum(0, a, 0.5, 0, at, -3.0)
        g.synchronize()
        want = vals[0] * 0.5 + -3.0 * bm.kat_transpose(bls[0], vals[0])
        assert np.array_equal(a.cpu().numpy(), want)
        g.matrix_sum(0, a, 2.0, 0, a, 0.25)                   # b is a: fl(2a), then fl(2a) + fl(0.25 fl(2a))
        g.synchronize()
        want = want * 2.0 + 0.25 * (want * 2.0)
        assert np.array_equal(a.cpu().numpy(), want)
        g.matrix_sum(1, b, 1.5, 0, at, 0.75)                  # the wider range keeps its other blocks
        g.synchronize()
        want_b, t = vals[1].copy(), bm.kat_transpose(bls[0], vals[0])
        for key, (off, ni, nj) in short.items():
            o = wide[key][0]
            want_b[o:o + ni * nj] = 1.5 * vals[1][o:o + ni * nj] + 0.75 * t[off:off + ni * nj]
        assert np.array_equal(b.cpu().numpy(), want_b)


def test_exact_sums_of_extreme_terms():
    """Traces with subnormal and huge terms, both signs, cancelling sums, zeros, infinities and NaN: the exact sum
    rounded once (Fractions of the rounded products; terms below 2^-150 of the largest do not occur)."""
    import fractions
    import torch
    import cq_b200
    g = cq_b200.System(*inputs.si_cluster(5, sigma=0.1, seed=71), np.full(5, 4, np.int32), [9.0])
    n = g.length(0)
    rng = np.random.default_rng(8)
    cases = [np.where(rng.random(n) < 0.5, 5e-324, -3e-310), rng.standard_normal(n) * 2.0 ** rng.integers(-40, 40, n),
             rng.standard_normal(n) * 1e300, np.zeros(n)]
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    for x in cases:
        d = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        want = float(sum((fractions.Fraction(float(v)) for v in x), fractions.Fraction(0)))
        assert g.product_trace(0, d, one) == want
        assert cq_b200.exact_dots_noalloc([d] * 3, [one, None, one]) == [want] * 3
    for bad in (np.inf, np.nan):
        d = torch.from_numpy(np.where(np.arange(n) == n - 1, bad, 1.0)).cuda()
        torch.cuda.synchronize()
        assert np.isnan(g.product_trace(0, d, one))
        assert g.product_trace(0, one, one) == n              # the flags of the last sum are cleared
