"""LinearBatch.solve reads its results back in a second library call: no other solve of the
same batch may be queued in between, whichever method queues it."""
import threading

import numpy as np

import rans_uq_b200.linear as lin


def test_no_solve_between_a_solve_and_its_results(monkeypatch):
    calls, inside, release = [], threading.Event(), threading.Event()

    def call(name, *args):
        calls.append((name, threading.current_thread().name))
        if name == "rq_linsys_solve_device" and threading.current_thread().name == "first":
            inside.set()
            release.wait(10)

    monkeypatch.setattr(lin.N, "call", call)
    batch = lin.LinearBatch([lin.LinearSystem.from_arrays(
        [2.0], [], [], [3.0], np.zeros(0, np.int32), np.zeros(0, np.int32))])
    first = threading.Thread(target=batch.solve, name="first")
    second = threading.Thread(target=batch.solve_device, args=(10, 1e-6), name="second")
    first.start()
    assert inside.wait(10)
    second.start()
    second.join(0.2)
    release.set()
    first.join(10)
    second.join(10)
    names = [c for c in calls if c[0] in ("rq_linsys_solve_device", "rq_linsys_results")]
    assert names == [("rq_linsys_solve_device", "first"), ("rq_linsys_results", "first"),
                     ("rq_linsys_solve_device", "second")]
