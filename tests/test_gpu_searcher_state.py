"""The Searcher's status and streams: a pass that reports an error raises from result() of that run alone, and an
exception while a run is queued leaves the caller's stream and device as they were."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def searcher(mini):
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import SearchParams
    l1, sp, _ = mini
    p = SearchParams(fragment_ppm=(-0.02, 0.02), fragment_unit="da", max_fragment_charge=1)
    gi = E.GpuIndex(l1, p, {"C": 57.021464}, {"M": 15.9949})
    return E, E.Searcher(gi, l1, p, depth=2), sp


@pytest.mark.parametrize("bits,text", [(1, "timed out"), (2, "bound was exceeded"), (4, "device status 4")])
def test_status_of_a_pass_is_raised(searcher, bits, text):
    E, se, sp = searcher
    want = se.search(sp)[0]
    a, b = se.submit(sp), se.submit(sp)
    a[1].done.synchronize()
    a[1].status.fill_(bits)           # what the first run's pass would have read back
    with pytest.raises(RuntimeError, match=text):
        se.result(a)
    assert se.result(b)[0].equals(want)


def test_exception_while_queueing_restores_the_stream(searcher, monkeypatch):
    import torch
    E, se, sp = searcher
    want = se.search(sp)[0]
    mine = torch.cuda.Stream()
    slot = se.slots[next(iter(se.slots))][se._turn[next(iter(se.slots))]]

    def fail():
        raise KeyboardInterrupt
    with torch.cuda.stream(mine):
        with monkeypatch.context() as m:
            m.setattr(slot.gp, "replay", fail)
            with pytest.raises(KeyboardInterrupt):
                se.submit(sp)
        assert torch.cuda.current_stream() == mine
    assert torch.cuda.current_stream() == torch.cuda.default_stream()
    slot.busy = False
    for _ in range(3):
        assert se.search(sp)[0].equals(want)
