"""Products at the edges of the staged kernels: every block size from 1 to 16, operands on an odd 8-byte boundary, pair
lists of 0, 1, 2 and a few terms (fewer than a kernel's stages or the four pairs of a tensor-core round), fused and split
arithmetic."""
import numpy as np
import pytest

import blockmaps as bm
from cq_b200 import inputs
from cq_oracle import OracleSystem

pytestmark = pytest.mark.gpu

# name -> (coordinates, block size of atom k)
SIZES = {"u1": ("cell2", lambda k: 1), "u3": ("cluster33", lambda k: 3), "u9": ("cell2", lambda k: 9),
         "u13": ("cluster33", lambda k: 13), "u16": ("cell2", lambda k: 16), "1to16": ("cell2", lambda k: 1 + k % 16),
         "1to3": ("cluster33", lambda k: 1 + k % 3), "4_13_many": ("cell3", lambda k: 13 if k % 3 == 0 else 4)}


def _system(sizes, rc):
    shape, nd = SIZES[sizes]
    if shape.startswith("cell"):
        coords, cell = inputs.diamond_si(int(shape[4:]), sigma=0.05, seed=41)
    else:
        coords, cell = inputs.si_cluster(int(shape[7:]), sigma=0.1, seed=42)
    return coords, cell, np.array([nd(k) for k in range(len(coords))], np.int32), rc


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("sizes", sorted(SIZES))
def test_fused_products_bits(sizes, mult_type):
    """FP64 with fused multiply-add: the tensor cores (FP64_TC, and FP64_FMA above 8 x 8), the group kernel and the generic
    one, alone and in a batch, with 16-byte aligned operands and on an odd multiple of 8 bytes: the bits of the oracle's
    default kernel with each multiply-add fused."""
    import torch
    import cq_b200
    sysargs = _system(sizes, [14.0, 6.0, 20.0] if mult_type == 2 else [6.0, 8.0, 14.0])
    coords, cell = sysargs[:2]
    o, g = OracleSystem(*sysargs), cq_b200.System(*sysargs)
    bls = [bm.oracle_blocklist(o, r, coords, cell) for r in range(3)]
    ops = [inputs.random_blocks(bls[r], 17 + r, inputs.TAG_RANDOM_A) for r in range(3)]
    out = 2 if mult_type == 1 else 0
    ref = [x.copy() for x in ops]
    ref[out][:] = 0.0
    o.mat_mult(mult_type, 0, 1, 2, *ref, kernel="default_fma")
    for shift in (0, 1):
        dev = []
        for r in range(3):
            t = torch.full((len(ops[r]) + 1,), float("nan"), dtype=torch.float64, device="cuda")
            if r != out:
                t[shift:shift + len(ops[r])] = torch.from_numpy(ops[r])
            dev.append(t[shift:shift + len(ops[r])])
        for prec, variant in ((cq_b200.PREC_FP64_TC, -1), (cq_b200.PREC_FP64_FMA, -1), (cq_b200.PREC_FP64_FMA, 4),
                              (cq_b200.PREC_FP64_FMA, 0), (cq_b200.PREC_FP64_FMA, None)):
            dev[out].fill_(float("nan"))
            torch.cuda.synchronize()
            if variant is None:
                g.set_mult_variant(-1)
                cq_b200.mat_mult_batch([(g, mult_type, 0, 1, 2, *dev, prec)])
            else:
                g.set_mult_variant(variant)
                g.mat_mult(mult_type, 0, 1, 2, *dev, precision=prec)
            g.synchronize()
            assert np.array_equal(dev[out].cpu().numpy(), ref[out]), (shift, prec, variant)


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("ncell", [2, 3])
def test_4x4_products_off_alignment(ncell, mult_type):
    """Uniform 4 x 4 blocks on an odd 8-byte boundary leave the 4 x 4 kernels (they read 16-byte vectors): few and many
    output blocks, both roundings, alone and in a batch."""
    import torch
    import cq_b200
    coords, cell = inputs.diamond_si(ncell, sigma=0.05, seed=41)
    sysargs = (coords, cell, np.full(len(coords), 4, np.int32), [14.0, 6.0, 20.0] if mult_type == 2 else [6.0, 8.0, 14.0])
    o, g = OracleSystem(*sysargs), cq_b200.System(*sysargs)
    bls = [bm.oracle_blocklist(o, r, coords, cell) for r in range(3)]
    ops = [inputs.random_blocks(bls[r], 27 + r, inputs.TAG_RANDOM_A) for r in range(3)]
    out = 2 if mult_type == 1 else 0
    for exact, kernel in ((True, "default"), (False, "default_fma")):
        ref = [x.copy() for x in ops]
        ref[out][:] = 0.0
        o.mat_mult(mult_type, 0, 1, 2, *ref, kernel=kernel)
        # one operand at a time off the boundary, then all of them
        for shifts in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)):
            dev = []
            for r in range(3):
                t = torch.full((len(ops[r]) + 1,), float("nan"), dtype=torch.float64, device="cuda")
                if r != out:
                    t[shifts[r]:shifts[r] + len(ops[r])] = torch.from_numpy(ops[r])
                dev.append(t[shifts[r]:shifts[r] + len(ops[r])])
            for batch in (False, True):
                dev[out].fill_(float("nan"))
                torch.cuda.synchronize()
                if batch:
                    cq_b200.mat_mult_batch([(g, mult_type, 0, 1, 2, *dev, int(exact))])
                else:
                    g.mat_mult(mult_type, 0, 1, 2, *dev, exact=exact)
                g.synchronize()
                assert np.array_equal(dev[out].cpu().numpy(), ref[out]), (exact, shifts, batch)


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("sizes", ["1to16", "1to3", "u13", "u16"])
@pytest.mark.parametrize("rc", [(5.0, 5.0, 12.0), (6.0, 8.0, 14.0)])
def test_split_kernels_ragged_sizes_and_short_lists(sizes, rc, mult_type):
    """The per-block split kernels on every block size and on lists of 0, 1 and 2 terms (the ring holds three): within
    2^-14 (two parts) and 2^-20 (three parts) of sum |a||b| per element, blocks without terms written as zeros."""
    import cq_b200
    rc = [rc[0], rc[1], rc[2], 24.0] if mult_type == 1 else [rc[2], rc[1], rc[0], 24.0]   # the last widens the cover only
    sysargs = _system(sizes, rc)
    coords, cell = sysargs[:2]
    o, g = OracleSystem(*sysargs), cq_b200.System(*sysargs)
    bls = [bm.oracle_blocklist(o, r, coords, cell) for r in range(3)]
    ops = [inputs.random_blocks(bls[r], 37 + r, inputs.TAG_RANDOM_A) for r in range(3)]
    out = 2 if mult_type == 1 else 0
    ref, bound = [x.copy() for x in ops], [np.abs(x) for x in ops]
    ref[out][:] = 0.0
    bound[out][:] = 0.0
    o.mat_mult(mult_type, 0, 1, 2, *ref)
    o.mat_mult(mult_type, 0, 1, 2, *bound)
    if rc[1] == 5.0:
        # terms per output block: the same product of a system with one orbital per atom, all elements 1
        o1 = OracleSystem(coords, cell, np.ones(len(coords), np.int32), rc)
        ones = [np.ones(o1.length(r)) for r in range(3)]
        ones[out][:] = 0.0
        o1.mat_mult(mult_type, 0, 1, 2, *ones)
        assert {0.0, 1.0, 2.0} <= set(ones[out])
    g.set_mixed_kernel(1)
    for prec, tol in ((cq_b200.PREC_BF16X3, 2.0 ** -14), (cq_b200.PREC_BF16X6, 2.0 ** -20)):
        got = [x.copy() for x in ops]
        got[out][:] = np.nan
        g.mat_mult_host(mult_type, 0, 1, 2, *got, precision=prec)
        assert not np.any(np.isnan(got[out]))
        err = np.abs(got[out] - ref[out])
        assert np.all(err <= tol * bound[out] + 1e-300), np.max(err / np.maximum(bound[out], 1e-300))
        assert err.max() > 0
        assert np.all(got[out][bound[out] == 0] == 0)


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("shape,n_out_range,sizes,variant", [
    ("few", (0, 2000), (1,), 0), ("few", (0, 2000), (1, 4), 0), ("few", (0, 2000), (5, 2), 0), ("few", (0, 2000), (8,), 0),
    ("few", (0, 2000), (6, 3), 0), ("few", (0, 2000), (9,), 4), ("some", (2000, 17000), (5,), 0), ("some", (2000, 17000), (4, 1), 0),
    ("some", (2000, 17000), (6,), 4), ("many", (17000, 10 ** 6), (3,), 4), ("many", (17000, 10 ** 6), (1, 4), 4)])
def test_small_blocks_kernel_choice_and_bits(shape, n_out_range, sizes, variant, mult_type):
    """Blocks of few rows: the generic kernel where there are few output blocks, the group kernel elsewhere, both with the
    bits of the oracle's default kernel (one, two and eight elements per lane of the generic one)."""
    import cq_b200
    coords, cell = {"few": lambda: inputs.si_cluster(24, sigma=0.1, seed=91), "some": lambda: inputs.diamond_si(2, sigma=0.05, seed=92),
                    "many": lambda: inputs.diamond_si(3, sigma=0.05, seed=93)}[shape]()
    nsf = np.array([sizes[k % len(sizes)] for k in range(len(coords))], np.int32)
    rc = [9.0, 6.0, 15.0] if mult_type == 1 else [15.0, 6.0, 21.0]
    o, g = OracleSystem(coords, cell, nsf, rc), cq_b200.System(coords, cell, nsf, rc)
    out = 2 if mult_type == 1 else 0
    assert n_out_range[0] <= g.n_blocks(out) < n_out_range[1]
    bls = [bm.oracle_blocklist(o, r, coords, cell) for r in range(3)]
    ops = [inputs.random_blocks(bls[r], 47 + r, inputs.TAG_RANDOM_A) for r in range(3)]
    ref, got = [x.copy() for x in ops], [x.copy() for x in ops]
    ref[out][:] = 0.0
    o.mat_mult(mult_type, 0, 1, 2, *ref)
    for v in (-1, 0, 4):
        g.set_mult_variant(v)
        got[out][:] = np.nan
        g.mat_mult_host(mult_type, 0, 1, 2, *got)
        assert np.array_equal(got[out], ref[out]), v
        assert g.product_tuning(mult_type, 0, 1, 2)[0] == variant


@pytest.mark.parametrize("sizes", ["u1", "u3", "u9", "u13", "u16", "1to16", "1to3"])
def test_transposes_of_every_block_size(sizes):
    """Transposes, staged and direct, against index arithmetic; transposing twice gives the matrix back."""
    import torch
    import cq_b200
    sysargs = _system(sizes, [7.0, 9.0])
    coords, cell = sysargs[:2]
    g = cq_b200.System(*sysargs)
    for r in range(2):
        bl = g.blocklist(r, coords, cell)
        v = inputs.random_blocks(bl, 57 + r, inputs.TAG_RANDOM_A)
        a = torch.from_numpy(v).cuda()
        at, back = torch.full_like(a, float("nan")), torch.full_like(a, float("nan"))
        torch.cuda.synchronize()
        g.transpose(r, a, at)
        g.transpose(r, at, back)
        g.synchronize()
        assert np.array_equal(at.cpu().numpy(), bm.kat_transpose(bl, v))
        assert torch.equal(back, a)


def test_row_kernel_builds_no_output_order():
    """The type-2 4 x 4 row kernel walks rows of B, not the output order: its first call launches one kernel."""
    import torch
    import cq_b200
    coords, cell = inputs.si_cluster(33, sigma=0.1, seed=95)
    g = cq_b200.System(coords, cell, np.full(len(coords), 4, np.int32), [10.0, 8.0, 18.0])
    ops = [torch.rand(g.length(r), dtype=torch.float64, device="cuda") for r in range(3)]
    torch.cuda.synchronize()
    g.product_work(2, 0, 1, 2)
    g.set_mult_variant(4)
    before = g.launch_count()
    g.mat_mult(2, 0, 1, 2, *ops)
    g.synchronize()
    assert g.launch_count() - before == 1


@pytest.mark.parametrize("tables", [("u4",), ("1_4",), ("u4", "1_4", "u13", "5_13", "u16", "u2"), ("u2", "u4")])
@pytest.mark.parametrize("exact", [True, False])
def test_batches_of_small_and_other_blocks(tables, exact):
    """Batches of 4 x 4 products alone (their own kernel), of small blocks alone and of every kind in one table, both mult
    types, few and many output blocks: the bits of the separate products."""
    import torch
    import cq_b200
    items, outs, keep = [], [], []
    gen = torch.Generator(device="cuda")
    gen.manual_seed(23)
    for k, name in enumerate(tables):
        sizes = [int(x) for x in name.lstrip("u").split("_")]
        for coords, cell in (inputs.si_cluster(21 + k, sigma=0.1, seed=97), inputs.diamond_si(2, sigma=0.05, seed=98)):
            nsf = np.array([sizes[i % len(sizes)] for i in range(len(coords))], np.int32)
            g = cq_b200.System(coords, cell, nsf, [7.0, 6.0, 13.0])
            keep.append(g)
            for t in (1, 2):
                ops = [torch.rand(g.length(r), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for r in range(3)]
                o = 2 if t == 1 else 0
                torch.cuda.synchronize()
                g.mat_mult(t, 0, 1, 2, *ops, exact=exact)
                g.synchronize()
                outs.append((ops[o], ops[o].clone()))
                ops[o].fill_(float("nan"))
                items.append((g, t, 0, 1, 2, *ops, int(exact)))
    torch.cuda.synchronize()
    cq_b200.mat_mult_batch(items)
    for g in keep:
        g.synchronize()
    for got, want in outs:
        assert torch.equal(got, want)
