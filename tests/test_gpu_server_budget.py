"""A server whose budget leaves no room for several guesses per slice decodes with one
(mmrecode_gb300/csrc/arena.h): every result equals the oracle's, with budgets from just above
what a request is reserved to plenty."""
import pytest

import mmrecode_gb300 as m
import oracle
from mmrecode_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sub,q,ri", [(1280, 720, "420", 97, 0), (320, 240, "420", 75, 0), (640, 480, "420", 80, 1)])
def test_results_do_not_depend_on_the_budget(w, h, sub, q, ri):
    packets = synth.mjpeg_stream(801, 4, w, h, sub, q, ri)
    refs = [oracle.jpeg_decode(p) for p in packets]
    planar = sum(pw * ph for pw, ph, _ in refs[0].frame.planes)
    one = 8 * max(map(len, packets)) + planar * 9 // 2 + 2 * planar + 65536  # what such a request is reserved
    for share in (one + 64, 4 * one, 64 * one):
        with m.Server(engines=1, max_batch=4, memory_budget=share) as srv:
            tickets = [srv.submit(p, m.CODEC_MJPEG, m.OUTPUT_PLANAR) for p in packets]
            for t, ref in zip(tickets, refs):
                r, payload, _ = srv.wait(t)
                assert r.status == ref.status == 0, r.message
                assert payload == b"".join(d for _, _, d in ref.frame.planes)
            assert srv.stats()["peak_budget_bytes"] <= share
