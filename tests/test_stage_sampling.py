"""Native completion of a step's sampling records against the same rule written out in Python."""
import struct

import numpy as np
import pytest

from ronn_b200.api.errors import SessionError
from ronn_b200.serving.scheduler import HostBatchBuffers, Scheduler

CAP = 256


@pytest.mark.parametrize("prompt_len,new", [(1, 0), (5, 3), (64, 1), (65, 2), (300, 4), (30, 260)])
def test_records_and_windows(prompt_len, new):
    sched = Scheduler(16, 200, 8, 2048, 0, "fcfs", False, 64)
    rng = np.random.default_rng(prompt_len)
    prompts = {7: rng.integers(0, 1000, prompt_len).tolist(), 9: [3, 4]}
    for rid, p in prompts.items():
        sched.add(rid, p, 300)
    host = HostBatchBuffers(2048, 8, 64, pin=False)
    out = {7: [], 9: []}
    for step in range(new):
        sb = sched.fill(host, sched.schedule())
        toks = rng.integers(0, 1000, sb.n_items).astype(np.int32)
        for rid, t in zip(sb.req_ids.tolist(), toks.tolist()):
            out[rid].append(t)
        sched.commit(toks)
    base = {7: -5, 9: 2 ** 63 + 12345}
    penalty = {7: 1.1, 9: 1.0}
    ids = np.array([9, 7], dtype=np.int64)
    rec = bytearray()
    for rid in ids.tolist():
        rec += struct.pack("<fffiQii", 0.8, 0.95, penalty[rid], 50, base[rid] & 0xFFFFFFFFFFFFFFFF, 99, 0)
    rec = np.frombuffer(bytes(rec), dtype=np.uint8).copy()
    recent = np.full((2, CAP), -1, dtype=np.int32)
    assert sched.stage_sampling(ids, rec.ctypes.data, recent.ctypes.data, CAP)
    for row, rid in enumerate(ids.tolist()):
        t, tp, rp, k, seed, n_recent, counter = struct.unpack_from("<fffiQii", rec, row * 32)
        assert seed == (base[rid] * 0x100000001B3 + len(out[rid])) & 0xFFFFFFFFFFFFFFFF and (k, counter) == (50, 0)
        window = (prompts[rid][-64:] + out[rid])[-CAP:] if penalty[rid] != 1.0 else []
        assert n_recent == len(window) and recent[row, :n_recent].tolist() == window and (recent[row, n_recent:] == -1).all()


def test_no_window_and_unknown_request():
    sched = Scheduler(16, 50, 4, 512, 0, "fcfs", False, 16)
    sched.add(1, [5, 6, 7], 4)
    rec = np.frombuffer(struct.pack("<fffiQii", 1.0, 1.0, 1.0, 0, 3, 0, 0), dtype=np.uint8).copy()
    recent = np.zeros((1, CAP), dtype=np.int32)
    assert not sched.stage_sampling(np.array([1]), rec.ctypes.data, recent.ctypes.data, CAP)
    with pytest.raises(SessionError):
        sched.stage_sampling(np.array([2]), rec.ctypes.data, recent.ctypes.data, CAP)
