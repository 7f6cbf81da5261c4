"""Downloads of one batch from several threads at once: every thread gets its
channel's fields, as one thread alone does (the calls share the batch's stream
and its staging buffer; the binding releases the interpreter lock in a call)."""
import threading

import numpy as np
import pytest

from lbm_mirror_gb300 import Batch
from lbm_mirror_gb300.workloads import batch_channels, channel_program

pytestmark = pytest.mark.gpu


def test_downloads_from_several_threads():
    channels = batch_channels(24, nx_range=(64, 300), ny_range=(32, 96))
    b = Batch(channels, channel_program(0.8))
    b.step(30)
    other = Batch(channels, channel_program(0.8))
    other.step(30)
    want = [(other.populations(c), *other.macros(c)) for c in range(other.n)]
    other.close()
    wrong = []
    gate = threading.Barrier(6)

    def reader(k):
        gate.wait()
        for i in range(60):
            c = (7 * k + i) % b.n
            got = b.populations(c) if (i + k) % 2 else b.macros(c)
            ref = want[c][0] if (i + k) % 2 else want[c][1:]
            same = np.array_equal(got, ref) if (i + k) % 2 else all(np.array_equal(x, y) for x, y in zip(got, ref))
            if not same:
                wrong.append((k, i, c))

    threads = [threading.Thread(target=reader, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    b.close()
    assert not wrong, wrong[:5]
