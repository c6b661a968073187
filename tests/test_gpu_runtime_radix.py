"""The runtime-radix kernel (csrc/rx_kernel.cuh) against the oracle: lengths
that have no compiled kernel, at the edges of its range -- every radix, primes
17..31 (alone, doubled and two of them), one-stage and long lengths (the
aliased staging area from about 4700 points), odd counts of lines, contiguous
and strided lines, direct, transposed and rank-split stores, every kind."""

import numpy as np
import pytest

import pencil_oracle as po
from pb_testutil import oracle_pencil

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pencil_b200 as pb  # noqa: E402
from pencil_b200 import _lib as L  # noqa: E402
from test_gpu_parity import CDT, RDT, check_transform, rand_field  # noqa: E402

R2R = ("DctI", "DctII", "DctIII", "DctIV", "DstI", "DstII", "DstIII", "DstIV", "Dht")
SHAPES = [((2, 2), (2, 3, 4)), ((2, 3), (11, 13, 26)), ((3, 2), (17, 34, 19)), ((1, 3), (31, 33, 29)),
          ((2, 2), (22, 23, 121)), ((2, 1), (143, 7, 286)), ((1, 2), (323, 5, 434)), ((2,), (1100, 9)),
          ((3,), (7, 2048 + 52)), ((2,), (4096, 3)), ((1,), (3, 5000)), ((1,), (6600, 2))]


@pytest.mark.parametrize("permute", [True, False])
@pytest.mark.parametrize("rb", [4, 8])
@pytest.mark.parametrize("dims,shape", SHAPES)
def test_complex_and_real_transforms(dims, shape, rb, permute):
    rng = np.random.default_rng(31)
    topo, lay = pb.MpiTopology(dims), pb.DistributedLayout(permute)
    plan = pb.C2cPlan.from_shape(topo, shape, (3,), layout=lay, dtype=CDT[rb])
    assert "runtime_radix" in plan.step_kernels(L.FORWARD) + plan.step_kernels(L.INVERSE)
    route = po.c2c_route(po.Topology(dims), shape, None, permute)
    x = rand_field(rng, shape, (3,), True, rb)
    for d in ("fwd", "inv", "bwd"):
        check_transform(plan, route, x, 3, rb, True, d)
    plan = pb.R2cPlan.from_shape(topo, shape, (3,), layout=lay, dtype=RDT[rb])
    route = po.r2c_route(po.Topology(dims), shape, None, permute)
    x = rand_field(rng, shape, (3,), False, rb)
    check_transform(plan, route, x, 3, rb, False, "fwd")
    spec = po.gather(oracle_pencil(plan.output_pencil),
                     po.execute_forward(route, po.scatter(oracle_pencil(plan.input_pencil), x, (3,))), (3,))
    for d in ("inv", "bwd"):
        check_transform(plan, route, spec, 3, rb, True, d)


@pytest.mark.parametrize("permute", [True, False])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("rb", [4, 8])
@pytest.mark.parametrize("kind", R2R)
def test_real_to_real_kinds(kind, rb, cplx, permute):
    rng = np.random.default_rng(32)
    for dims, shape in (((2, 3), (13, 22, 9)), ((1, 2), (5, 33, 286)), ((2,), (1024, 3))):
        plan = pb.R2rPlan.from_shape(pb.MpiTopology(dims), shape, (3,), [kind] * len(shape),
                                     layout=pb.DistributedLayout(permute), dtype=CDT[rb] if cplx else RDT[rb])
        assert "runtime_radix" in plan.step_kernels(L.FORWARD)
        route = po.r2r_route(po.Topology(dims), shape, [kind] * len(shape), permute)
        x = rand_field(rng, shape, (3,), cplx, rb)
        for d in ("fwd", "inv", "bwd"):
            check_transform(plan, route, x, 3, rb, cplx, d)


@pytest.mark.parametrize("make", ["r2c", "DctI", "DctII", "DctIII", "DstII", "DstIII", "DstIV"])
def test_adjoint_weights(make):
    """<A x, y> = <x, A^T y> in f64 for the weighted kinds."""
    torch.manual_seed(33)
    topo, shape = pb.MpiTopology((2, 2)), (13, 22, 26)
    if make == "r2c":
        plan = pb.R2cPlan.from_shape(topo, shape, (), dtype=torch.float64)
    else:
        plan = pb.R2rPlan.from_shape(topo, shape, (), [make] * 3, dtype=torch.float64)
    x = torch.randn(plan.info.input_elems, dtype=plan.input_dtype, device="cuda")
    y = torch.randn(plan.info.output_elems, dtype=plan.output_dtype, device="cuda")
    ax, aty = plan.allocate_output(), plan.allocate_input()
    plan.forward(x, ax)
    plan.vjp_forward(y, aty)
    lhs, rhs = float(torch.sum((ax.conj() * y).real)), float(torch.sum(x * aty))
    assert abs(lhs - rhs) <= 1e-12 * float(torch.linalg.vector_norm(ax) * torch.linalg.vector_norm(y))


@pytest.mark.parametrize("permute", [True, False])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("rb", [4, 8])
@pytest.mark.parametrize("shape,kinds", [((34, 62, 48), ("DstI",) * 3), ((36, 64, 106), ("DctI",) * 3),
                                         ((100, 22, 340), ("DstI",) * 3), ((4, 90, 12), ("DctI",) * 3),
                                         ((10, 384, 6), ("DstI", "DstI", "DctI"))])
def test_type_one_kinds_with_odd_n(shape, kinds, rb, cplx, permute):
    """Type-I kinds whose symmetric extension has 2N points, N odd: the N-point
    form on the compiled and the runtime-radix kernel, Bluestein included."""
    rng = np.random.default_rng(34)
    plan = pb.R2rPlan.from_shape(pb.MpiTopology((2, 3)), shape, (3,), kinds, layout=pb.DistributedLayout(permute),
                                 dtype=CDT[rb] if cplx else RDT[rb])
    route = po.r2r_route(po.Topology((2, 3)), shape, list(kinds), permute)
    x = rand_field(rng, shape, (3,), cplx, rb)
    for d in ("fwd", "inv", "bwd"):
        check_transform(plan, route, x, 3, rb, cplx, d)
