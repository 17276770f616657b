"""The chained per-loop entry points behind whatever else a stream holds: copies,
clears, events of other streams, and in captured graphs (GPU)."""
import numpy as np
import pytest

from mgcfd import ops

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = 70_001


def _arrays():
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    rnd = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    return dict(sf=rnd(N), flux=rnd(N, 5), old=rnd(N, 5), var=rnd(N, 5), res=rnd(N, 5), rms=torch.zeros(1, dtype=torch.float64, device="cuda"),
                src=rnd(N, 5), extra=rnd(N, 5))


def _program(a, main, side, between):
    """copy -> (something else) -> time_step -> (something else) -> residual -> rms."""
    s = main.cuda_stream

    def something():
        if between == "copy":
            a["flux"].copy_(a["src"])
        elif between == "clear":
            a["flux"].zero_()
        elif between == "join":
            event = torch.cuda.Event()
            event.record(main)
            with torch.cuda.stream(side):
                side.wait_event(event)
                a["flux"].add_(a["extra"])
                done = torch.cuda.Event()
                done.record(side)
            main.wait_event(done)

    with torch.cuda.stream(main):
        ops.copy_double(N, a["var"].data_ptr(), a["old"].data_ptr(), s)
        something()
        ops.time_step(N, 1, a["sf"].data_ptr(), a["flux"].data_ptr(), a["old"].data_ptr(), a["var"].data_ptr(), s)
        something()
        ops.residual(N, a["old"].data_ptr(), a["var"].data_ptr(), a["res"].data_ptr(), s)
        a["rms"].zero_()
        ops.calc_rms(N, a["res"].data_ptr(), a["rms"].data_ptr(), s)


def _expected(a, between, times):
    v = {k: x.cpu().numpy().copy() for k, x in a.items()}

    def something():
        if between == "copy":
            v["flux"][:] = v["src"]
        elif between == "clear":
            v["flux"][:] = 0.0
        elif between == "join":
            v["flux"] += v["extra"]

    for _ in range(times):
        v["old"] = v["var"].copy()
        something()
        v["var"] = v["old"] + (v["sf"] * (1.0 / 3.0))[:, None] * v["flux"]
        v["flux"][:] = 0.0  # (the loop clears the increments it has used)
        something()
        v["res"] = v["var"] - v["old"]
    return v


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("between", ["nothing", "copy", "clear", "join"])
def test_chained_loops_follow_other_work(between, captured):
    a = _arrays()
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    want = _expected(a, between, 2)
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            _program(a, torch.cuda.current_stream(), side, between)
        for _ in range(2):
            graph.replay()
    else:
        for _ in range(2):
            _program(a, main, side, between)
    torch.cuda.synchronize()
    for k in ("old", "var", "res", "flux"):
        np.testing.assert_allclose(a[k].cpu().numpy(), want[k], rtol=0, atol=2.0 ** -50 * np.abs(want["var"]).max(), err_msg=k)
    assert a["rms"].item() == pytest.approx((want["res"] ** 2).sum(), rel=1e-12)
