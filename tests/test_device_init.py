"""Table uploads are ordered before every caller's first kernel.

The NTT and hash tables, a batched plan's descriptors and an instruction table go up with copies from pageable
memory on the legacy stream, which may return before the device has the words, while commits run on non-blocking
streams that the legacy stream does not order.  So each upload has to wait for its copies.  The window is
microseconds wide and no run can be made to fall into it, so the order of the calls is read from the source.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pil2-proofman_b200", "csrc")


def function_body(name, file="pil2_b200.cu"):
    src = open(os.path.join(CSRC, file)).read()
    src = re.sub(r"//[^\n]*", "", src)
    start = src.index("{", src.index(name + "("))
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


def test_batch_and_instruction_tables_are_waited_for():
    for body, copy in ((function_body("cudaError_t upload", "batch.cuh"), "cudaMemcpy(d_table"),
                       (function_body("void register_instruction_table"), "cudaMemcpy(a.d_table")):
        assert body.index(copy) < body.index("cudaStreamSynchronize(cudaStreamLegacy)")
