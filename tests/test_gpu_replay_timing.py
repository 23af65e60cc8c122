"""GPU times of replayed batches: every event keeps its own, however many replays follow and whatever becomes of the batch."""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu
pkg = load_pkg()
rt = pkg.runtime


@pytest.mark.parametrize("replays", [1, 64, 1022, 1023, 1024, 2500])
def test_every_replay_keeps_its_gpu_time(replays):
    ctx = rt.init()
    n = 1 << 18
    a, b, d = (ctx.buffer(data=np.full(n, v, np.float32)) for v in (1.0, 2.0, 0.0))
    batches = []
    for k in (1, 24):       # a short one and one that takes several times as long
        batch = ctx.batch(32)
        for _ in range(k):
            batch.dispatch(ctx.kernel("ameva_add_f32"), [a, b, d], [1, n, 1])
        batch.instantiate()
        batches.append(batch)
    events = [[batches[i].replay() for _ in range(replays)] for i in (0, 1)]
    for evs in events:
        evs[-1].wait()
    short = [0.0] * replays
    for i, ev in enumerate(events[0]):
        ev.wait()
        short[i] = ev.gpu_duration_us()
    for batch in batches:
        batch.destroy()     # the times of the second batch are read after it is gone
    for i, ev in enumerate(events[1]):
        ev.wait()
        us = ev.gpu_duration_us()
        assert 0 < short[i] < 1e6 and 0 < us < 1e6
        assert us == ev.gpu_duration_us()
    times = [ev.gpu_duration_us() for ev in events[1]]
    assert np.median(short) < np.median(times)
    for evs in events:
        for ev in evs:
            ev.destroy()
    for x in (a, b, d):
        x.destroy()
    ctx.destroy()


def test_more_replayable_batches_than_rings():
    ctx = rt.init()
    x = ctx.buffer(data=np.ones(1024, np.float32))
    batches = []
    for _ in range(70):
        batch = ctx.batch(1)
        batch.dispatch(ctx.kernel("ameva_add_f32"), [x, x, x], [1, 1024, 1])
        batch.instantiate()
        batches.append(batch)
    for batch in batches:
        ev = batch.replay()
        ev.wait()
        assert 0 < ev.gpu_duration_us() < 1e6
        ev.destroy()
    for batch in batches:
        batch.destroy()
    again = ctx.batch(1)
    again.dispatch(ctx.kernel("ameva_add_f32"), [x, x, x], [1, 1024, 1])
    again.instantiate()
    ev = again.replay()
    ev.wait()
    assert ev.gpu_duration_us() > 0
    ev.destroy()
    again.destroy()
    x.destroy()
    ctx.destroy()


def test_events_timed_and_destroyed_on_another_thread():
    """One thread replays and destroys the batch, another waits for the events, asks for their times and destroys them."""
    import queue
    import threading
    ctx = rt.init()
    n = 1 << 14
    x = ctx.buffer(data=np.ones(n, np.float32))
    todo, times, errors = queue.SimpleQueue(), [], []

    def drain():
        try:
            while (ev := todo.get()) is not None:
                ev.wait()
                if len(times) % 3:          # (some are destroyed without a look at their time)
                    times.append(ev.gpu_duration_us())
                else:
                    times.append(1.0)
                ev.destroy()
        except Exception as e:              # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    worker = threading.Thread(target=drain)
    worker.start()
    replays = 0
    for _ in range(3):
        batch = ctx.batch(4)
        for _ in range(2):
            batch.dispatch(ctx.kernel("ameva_add_f32"), [x, x, x], [1, n, 1])
        batch.instantiate()
        for _ in range(1500):
            todo.put(batch.replay())
            replays += 1
        batch.destroy()                     # the worker still holds events of it
    todo.put(None)
    worker.join(60)
    assert not worker.is_alive() and not errors
    assert len(times) == replays and all(0 < t < 1e6 for t in times)
    x.destroy()
    ctx.destroy()
