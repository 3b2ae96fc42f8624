"""Products captured into a caller's CUDA graph on a system whose pair lists exist but whose staged kernels have not run
yet: what those kernels build on their first use (which allocates and waits) cannot be built inside a capture, so the
launch has to do without it, with the same results."""
import numpy as np
import pytest

from cq_b200 import inputs

pytestmark = pytest.mark.gpu

SIZES = {"u13": lambda k: 13, "4_13": lambda k: 13 if k % 3 == 0 else 4, "u4": lambda k: 4}


@pytest.mark.parametrize("mult_type", [1, 2])
@pytest.mark.parametrize("sizes,precision,variant,batch", [
    ("u13", "PREC_FP64_TC", -1, False), ("4_13", "PREC_FP64_FMA", -1, False), ("u13", "PREC_FP64", 4, False),
    ("4_13", "PREC_FP64", 4, True), ("u4", "PREC_FP64", 4, False), ("u4", "PREC_FP64", 5, False), ("u4", "PREC_FP64", -1, False),
    ("u4", "PREC_FP64_FMA", 6, False), ("u4", "PREC_FP64", -1, True)])
def test_first_call_inside_a_capture(sizes, precision, variant, batch, mult_type):
    import torch
    import cq_b200
    prec = getattr(cq_b200, precision)
    coords, cell = inputs.si_cluster(37, sigma=0.1, seed=81)
    nsf = np.array([SIZES[sizes](k) for k in range(len(coords))], np.int32)
    outs = []
    for captured in (False, True):
        g = cq_b200.System(coords, cell, nsf, [8.0, 9.0, 17.0])
        g.set_mult_variant(variant)
        stream = torch.cuda.Stream()
        g.set_stream(stream.cuda_stream)
        g.product_work(mult_type, 0, 1, 2)                    # the pair lists
        gen = torch.Generator(device="cuda")
        gen.manual_seed(17)
        ops = [torch.rand(g.length(r), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for r in range(3)]
        out = ops[2 if mult_type == 1 else 0]
        out.fill_(float("nan"))
        torch.cuda.synchronize()

        def call():
            if batch:
                cq_b200.mat_mult_batch([(g, mult_type, 0, 1, 2, *ops, prec)])
            else:
                g.mat_mult(mult_type, 0, 1, 2, *ops, precision=prec)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                call()
            assert torch.isnan(out).all()                     # captured, not run
            graph.replay()
            torch.cuda.synchronize()
            first = out.clone()
            out.fill_(float("nan"))
            torch.cuda.synchronize()
            call()                                            # a direct call afterwards builds and uses them
            g.synchronize()
            assert torch.equal(out, first)
        else:
            call()
            g.synchronize()
        outs.append(out.clone())
        g.close()
    assert not torch.isnan(outs[0]).any()
    assert torch.equal(outs[0], outs[1])


def test_two_part_split_captured_before_its_kernel_is_chosen():
    """A two-part split product whose fragments and lists exist (from a three-part call) but whose kernel has not been chosen:
    the captured call runs on the blocks, a later direct one chooses (tiles, on this dense cluster)."""
    import torch
    import cq_b200
    coords, cell = inputs.si_cluster(100, sigma=0.1, seed=2, vacuum=15.0)
    g = cq_b200.System(coords, cell, np.full(len(coords), 13, np.int32), [20.0, 20.0, 40.0])
    stream = torch.cuda.Stream()
    g.set_stream(stream.cuda_stream)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(19)
    ops = [torch.rand(g.length(r), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for r in range(3)]
    torch.cuda.synchronize()
    g.mat_mult(1, 0, 1, 2, *ops, precision=cq_b200.PREC_BF16X6)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        g.mat_mult(1, 0, 1, 2, *ops, precision=cq_b200.PREC_BF16X3)
    ops[2].fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    captured = ops[2].clone()
    outs = {}
    for k in (-1, 0, 1):
        g.set_mixed_kernel(k)
        g.mat_mult(1, 0, 1, 2, *ops, precision=cq_b200.PREC_BF16X3)
        g.synchronize()
        outs[k] = ops[2].clone()
    assert torch.equal(captured, outs[1]) and torch.equal(outs[-1], outs[0]) and not torch.equal(outs[0], outs[1])
