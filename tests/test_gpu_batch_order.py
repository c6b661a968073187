"""Branch mode with plans that share buffers, one batch run by two threads, and
what a first execution creates."""

import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pencil_b200 as pb  # noqa: E402

SHAPES = [(96, 80, 64), (64, 96, 80), (48, 45, 50)]


def make_plans(shapes):
    return [pb.C2cPlan.from_shape(pb.MpiTopology((1, 2)), s, (2,), dtype=torch.complex64) for s in shapes]


def field(plan):
    return torch.randn(plan.info.input_elems, dtype=torch.complex64, device="cuda")


def run(batch, buffers, ws, stream):
    with torch.cuda.stream(stream if stream is not None else torch.cuda.default_stream()):
        batch.execute(buffers, ws, stream)
        batch.status(ws, stream)


@pytest.mark.parametrize("side_stream", [False, True])
def test_a_plan_reads_what_another_one_writes(side_stream):
    torch.manual_seed(51)
    plans = make_plans([SHAPES[0]] * 3)
    x, y, z, w = (field(plans[0]) for _ in range(4))
    ref = [x]
    for p in plans:
        ref.append(p.allocate_output())
        p.forward(ref[-2], ref[-1])
    batch = pb.PlanBatch(plans, ("forward",), autotune=False)
    ws = batch.allocate_workspace()
    stream = torch.cuda.Stream() if side_stream else None
    torch.cuda.synchronize()
    for _ in range(3):
        run(batch, [[x, y, z], [y, z, w]], ws, stream)
        assert torch.equal(w, ref[3]) and torch.equal(z, ref[2])
        y.zero_(), z.zero_(), w.zero_()
        torch.cuda.synchronize()


@pytest.mark.parametrize("side_stream", [False, True])
def test_plans_share_a_spectrum(side_stream):
    """One array for every plan's spectrum (the second plan's overlaps the
    first one's in part only)."""
    torch.manual_seed(52)
    plans = make_plans(SHAPES)
    xs = [field(p) for p in plans]
    pool = torch.zeros(max(p.info.output_elems for p in plans) + 64, dtype=torch.complex64, device="cuda")
    spectra = [pool[64 * (i == 1):][:p.info.output_elems] for i, p in enumerate(plans)]
    refs = []
    for p, x in zip(plans, xs):
        m, back = p.allocate_output(), p.allocate_input()
        p.forward(x, m)
        p.inverse(m, back)
        refs.append(back)
    batch = pb.PlanBatch(plans, autotune=False)
    ws = batch.allocate_workspace()
    back = [torch.zeros_like(x) for x in xs]
    torch.cuda.synchronize()
    run(batch, [xs, spectra, back], ws, torch.cuda.Stream() if side_stream else None)
    assert all(torch.equal(b, r) for b, r in zip(back, refs))


def test_a_shared_input_and_adjacent_outputs():
    """Plans that only read the same array, and outputs side by side in one."""
    torch.manual_seed(53)
    plans = make_plans([SHAPES[2]] * 4)
    x = field(plans[0])
    ref = plans[0].allocate_output()
    plans[0].forward(x, ref)
    out = torch.zeros(4 * ref.numel(), dtype=torch.complex64, device="cuda")
    batch = pb.PlanBatch(plans, ("forward",), autotune=False)
    ws = batch.allocate_workspace()
    run(batch, [[x] * 4, list(out.split(ref.numel()))], ws, None)
    assert all(torch.equal(o, ref) for o in out.split(ref.numel()))


@pytest.mark.parametrize("side_stream", [False, True])
def test_two_threads_run_one_batch(side_stream):
    torch.manual_seed(54)
    plans = make_plans(SHAPES)
    batch = pb.PlanBatch(plans, ("forward",), autotune=False)
    work, errors = [], []
    for _ in range(2):
        xs = [field(p) for p in plans]
        refs = []
        for p, x in zip(plans, xs):
            refs.append(p.allocate_output())
            p.forward(x, refs[-1])
        outs = [torch.zeros_like(r) for r in refs]
        work.append((xs, outs, refs, batch.allocate_workspace(), torch.cuda.Stream() if side_stream else None))
    torch.cuda.synchronize()

    def body(xs, outs, refs, ws, stream):
        try:
            for _ in range(20):
                run(batch, [xs, outs], ws, stream)
                if not all(torch.equal(o, r) for o, r in zip(outs, refs)):
                    errors.append("result")
                with torch.cuda.stream(stream if stream is not None else torch.cuda.default_stream()):
                    for o in outs:
                        o.zero_()
        except Exception as e:  # pragma: no cover
            errors.append(repr(e))

    threads = [threading.Thread(target=body, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []


def stream_ids(count):
    """Ids of newly made streams: consecutive where nobody else makes one."""
    cu, ids = C.CDLL("libcuda.so.1"), []
    for _ in range(count):
        st, i = C.c_void_p(), C.c_uint64()
        assert cu.cuStreamCreate(C.byref(st), 1) == 0
        assert cu.cuStreamGetId(st, C.byref(i)) == 0
        assert cu.cuStreamDestroy_v2(st) == 0
        ids.append(i.value)
    return ids


def test_a_first_execution_makes_no_streams():
    plans = make_plans(SHAPES)
    xs = [field(p) for p in plans]
    outs = [p.allocate_output() for p in plans]
    for p, x, o in zip(plans, xs, outs):
        p.forward(x, o)
    batch = pb.PlanBatch(plans, ("forward",), autotune=False)
    ws = batch.allocate_workspace()
    torch.cuda.synchronize()
    a, b, c = stream_ids(3)
    assert c - b == b - a
    run(batch, [xs, outs], ws, None)
    (d,) = stream_ids(1)
    assert d - c == b - a
    batch.set_mode("branches", 5)  # made here
    (e,) = stream_ids(1)
    run(batch, [xs, outs], batch.allocate_workspace(), None)
    (f,) = stream_ids(1)
    assert e - d > b - a and f - e == b - a
