"""Round-trip errors of the runtime-radix kernel against the error of the
generic kernel's schedule (radices up to 8, constants rounded once) on the same
axis: forward and inverse of an n x 2 field of normal samples.  The second
columns are that schedule's relative L2 errors as measured on a B200; errors of
this many samples scatter by about 1%, so 5% more is a loss of accuracy."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pencil_b200 as pb  # noqa: E402


def round_trip_error(make, n, dtype):
    gen = torch.Generator(device="cuda").manual_seed(3)
    total = err = 0.0
    plan = make(n, dtype)
    for _ in range(1 + 2 ** 16 // (128 * n)):
        x = torch.randn(plan.info.input_elems, dtype=dtype, device="cuda", generator=gen)
        y, z = plan.allocate_output(), plan.allocate_input()
        plan.forward(x, y)
        plan.inverse(y, z)
        err += float(torch.linalg.vector_norm(z - x)) ** 2
        total += float(torch.linalg.vector_norm(x)) ** 2
    return (err / total) ** 0.5


def c2c(n, dtype):
    return pb.C2cPlan.from_shape(pb.MpiTopology((1,)), (n, 2), (64,), dtype=dtype)


def r2r(kind):
    return lambda n, dtype: pb.R2rPlan.from_shape(pb.MpiTopology((1,)), (n, 2), (64,), [kind, "Dht"], dtype=dtype)


@pytest.mark.parametrize("make,n,dtype,generic", [
    # composite radices: the rotations inside the butterflies
    (c2c, 2048, torch.complex64, 1.685e-7), (c2c, 3000, torch.complex64, 1.816e-7),
    (c2c, 4096, torch.complex64, 1.750e-7), (c2c, 1296, torch.complex128, 3.784e-16),
    # Bluestein's convolution lengths above 1024
    (c2c, 521, torch.complex64, 2.236e-7), (c2c, 521, torch.complex128, 4.078e-16),
    (c2c, 751, torch.complex64, 2.575e-7), (c2c, 1321, torch.complex64, 2.462e-7),
    # a type-I kind whose N-point form would take a shorter convolution
    (r2r("DstI"), 286, torch.float32, 2.198e-7),
    (r2r("DctII"), 41, torch.float64, 3.784e-16), (r2r("DctII"), 131, torch.float64, 4.399e-16),
])
def test_round_trip_error(make, n, dtype, generic):
    assert round_trip_error(make, n, dtype) <= 1.05 * generic
