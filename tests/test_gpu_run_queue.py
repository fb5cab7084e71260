"""run() on a queue of its own beside work on the current stream: the second copies of the path come from
memory that the current stream has freed but still reads and writes."""
import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPE = (40, 36, 33)


def _kw():
    rng = numpy.random.default_rng(5)
    return dict(epsilon=[rng.uniform(1, 4, SHAPE).astype(numpy.float32) for _ in range(3)],
                pmls=[{"axis": a, "polarity": p, "thickness": 4} for a in "xyz" for p in "np"],
                initial_fields={k: [rng.standard_normal(SHAPE).astype(numpy.float32) for _ in range(3)] for k in "EH"})


@pytest.mark.parametrize("path", ["hs", "ahead", "fused"])
@pytest.mark.parametrize("poynting", [True, False])
def test_copies_beside_work_on_the_current_stream(path, poynting):
    from opencl_fdtd_gb300 import Simulation
    if path == "hs" and not poynting:
        pytest.skip("the path needs Poynting")
    ref = Simulation(do_poynting=poynting, **_kw())
    ref.run(6, path="plain")
    queue = torch.cuda.Stream()
    sim = Simulation(do_poynting=poynting, queue=queue, **_kw())
    queue.wait_stream(torch.cuda.current_stream())
    queue.synchronize()
    blocks = [torch.empty_like(sim.E) for _ in range(2)]
    torch.cuda._sleep(20_000_000)                            # about 10 ms of the current stream
    for b in blocks:
        b.fill_(7.0)                                         # after the sleep
    del b, blocks                                            # free for the current stream, still to be written
    sim.run(6, path=path)
    queue.synchronize()
    torch.cuda.synchronize()
    for k in ("E", "H") + (("S",) if poynting else ()):
        assert torch.equal(getattr(ref, k), getattr(sim, k)), k
