"""The per-device initialisation orders its table uploads before every caller's first kernel.

The tables go up with copies from pageable memory on the legacy stream, which may return before the device has the
words, while commits run on non-blocking streams that the legacy stream does not order.  So the initialisation has to
wait for the copies before it marks the device ready.  The window is microseconds wide and no run can be made to fall
into it, so the order of the calls is read from the source.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pil2-proofman_b200", "csrc")


def function_body(name):
    src = open(os.path.join(CSRC, "pil2_b200.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    start = src.index("{", src.index(name + "()"))
    depth = 0
    for i in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[start:i + 1]
    raise AssertionError("unterminated function " + name)


def test_uploads_are_waited_for_before_the_device_is_ready():
    body = function_body("static int ensure_init_current")
    uploads = [body.index(call) for call in ("ntt::init_tables()", "merkle::init()")]
    wait = body.index("cudaStreamSynchronize(cudaStreamLegacy)")
    ready = body.index("g_init_done[dev] = true")
    assert max(uploads) < wait < ready
