"""Which kernel and FFT length the real-to-real kinds get: step_configs of the
first axis of an n x 4 field."""

import numpy as np
import pytest

import pencil_oracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pencil_b200 as pb  # noqa: E402
from pencil_b200 import _lib as L  # noqa: E402
from test_gpu_parity import check_transform, rand_field  # noqa: E402


def r2r_plan(kind, n, dtype):
    return pb.R2rPlan.from_shape(pb.MpiTopology((1,)), (n, 4), (3,), [kind, "Dht"], dtype=dtype)


@pytest.mark.parametrize("kind,n,dtype,kernel,fft_len", [
    # type I, 2N-point form: where the N-point one saves nothing or has no kernel
    ("DstI", 384, torch.float32, "mixed_radix", 770), ("DstI", 384, torch.float64, "mixed_radix", 770),
    ("DstI", 384, torch.complex64, "mixed_radix", 770), ("DctI", 106, torch.float64, "mixed_radix", 210),
    ("DstI", 124, torch.float32, "mixed_radix", 250),
    # N-point form: fewer stages in f64, radix 14 or 15 avoided in f32, runtime radices
    ("DstI", 124, torch.float64, "mixed_radix", 125), ("DctI", 106, torch.float32, "mixed_radix", 105),
    ("DstI", 350, torch.float32, "runtime_radix", 351), ("DctI", 456, torch.float64, "runtime_radix", 455),
    # Bluestein: the N-point form unless its convolution is the relatively shorter one
    ("DstI", 100, torch.float32, "bluestein", 101), ("DstI", 286, torch.float32, "bluestein", 574),
])
def test_kernel_and_length(kind, n, dtype, kernel, fft_len):
    c = r2r_plan(kind, n, dtype).step_configs(L.FORWARD)[-1]
    assert (c["kernel"], c["fft_len"]) == (kernel, fft_len)


@pytest.mark.parametrize("kind", ["DctIV", "DstIV"])
@pytest.mark.parametrize("rb,dtype", [(4, torch.float32), (8, torch.float64)])
def test_type_four_longer_than_the_row_tables(kind, rb, dtype):
    """A 770-point FFT with 1540 outputs per line, more than the compiled
    kernel's row tables hold: the runtime-radix kernel's."""
    plan = r2r_plan(kind, 1540, dtype)
    c = plan.step_configs(L.FORWARD)[-1]
    assert (c["kernel"], c["fft_len"]) == ("runtime_radix", 770)
    route = po.r2r_route(po.Topology((1,)), (1540, 4), [kind, "Dht"], True)
    x = rand_field(np.random.default_rng(35), (1540, 4), (3,), False, rb)
    for d in ("fwd", "inv", "bwd"):
        check_transform(plan, route, x, 3, rb, False, d)


@pytest.mark.parametrize("make,n,dtype,radices", [
    (pb.C2cPlan, 4096, torch.complex64, [16, 16, 16]), (pb.C2cPlan, 255, torch.complex128, [15, 17]),
    # Bluestein: 576 and 1024 points on the mixed-radix kernel, 2048 and 224 on the runtime-radix one
    (pb.C2cPlan, 257, torch.complex64, [3, 3, 8, 8]), (pb.C2cPlan, 509, torch.complex64, [2, 8, 8, 8]),
    (pb.C2cPlan, 521, torch.complex64, [4, 8, 8, 8]), ("DstI", 100, torch.float32, [4, 7, 8]),
])
def test_reported_radices(make, n, dtype, radices):
    """The stages of a pass; of a Bluestein pass the factors of its convolution
    length."""
    if isinstance(make, str):
        plan = r2r_plan(make, n, dtype)
    else:
        plan = make.from_shape(pb.MpiTopology((1,)), (n, 4), (3,), dtype=dtype)
    c = plan.step_configs(L.FORWARD)[-1]
    assert sorted(c["radices"]) == radices and (c["kernel"] == "bluestein") == (n not in (255, 4096))
