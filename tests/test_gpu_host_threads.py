"""The host threads that gather row-pointer batches (HostWorkers in csrc/model.cu): after a
gather one of them looks for the next one for 200 us, the others sleep."""
import os
import time

import pytest

import configs
import dlb200
import util

pytestmark = pytest.mark.gpu


@pytest.mark.skipif((os.cpu_count() or 1) < 8, reason="fewer host threads than the model keeps")
def test_one_worker_polls(gpu_ctx):
    rows = 1024
    cfg = configs.deep_brn_mlp(512, 64, 1, 8, rows, dropout=None)  # 2 MB of inputs
    X, _ = configs.synthetic_batch(cfg)
    model = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
    model.train_begin(rows)
    gathers = 100

    def workers_time(pause):
        """Processor time of the other threads, per gather."""
        start = time.process_time() - time.thread_time()
        for _ in range(gathers):
            model.forward_pass(rows, X)
            gpu_ctx.sync()
            time.sleep(pause)
        return (time.process_time() - time.thread_time() - start) / gathers

    workers_time(0.002)
    # Seven workers that all look take 1.4 ms; one takes 0.2, and the copying of 2 MB
    # at 2 GB/s a thread at most one more half.
    assert workers_time(0.002) < 0.9e-3
