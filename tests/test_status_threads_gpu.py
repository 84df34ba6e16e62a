"""Reading the device status from one thread while another keeps calling: the word that a call replaces may belong to
Python, and letting go of it must not wait for the interpreter while the reader waits for the word."""

import threading

import pytest
import torch

from delta_feedback_experiment_b200 import _lib, ops
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu


def test_status_is_read_while_another_thread_calls():
    d = make_inputs(1, 64, 1, 128, seed=1)
    args = [d[n].cuda() for n in INPUT_NAMES]
    done = threading.Event()
    ops.track_device_status(True)

    def call():
        for _ in range(300):
            ops.chunk_forward(*args, 128 ** -0.5, 1.5, 1e-6)
        done.set()

    def read():
        while not done.is_set():
            _lib.native().last_status(False)

    threads = [threading.Thread(target=f, daemon=True) for f in (call, read)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=60)
    assert done.is_set() and not any(t.is_alive() for t in threads)
    torch.cuda.synchronize()
    assert ops.last_device_status() == 0
