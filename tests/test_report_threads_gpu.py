"""Two threads read an engine's report on two streams: the one on the idle stream
does not wait for the other's."""
import threading
import time

import pytest

from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_a_report_waits_for_its_own_stream_only():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine

    b = scenes.building()
    eng = Engine(b["entries"], node_capacity=1 << 16, max_terminals=1 << 16)
    _, n, _ = eng.execute(b["axioms"], capacity=1 << 16)
    busy, idle = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    reports = []
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1_500_000_000)  # 0.7 s or more of an idle loop
    waiting = threading.Thread(target=lambda: reports.append(eng.report(busy)))
    waiting.start()
    time.sleep(0.1)  # into its wait
    got = eng.report(idle)
    still = not busy.query()
    waiting.join()
    torch.cuda.synchronize()
    eng.release()
    assert still and got["terminals"] == n and reports[0] == got
