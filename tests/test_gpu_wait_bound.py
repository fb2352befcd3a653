"""A tensor core product that does not complete within its bounded wait.

The probe runs the hashing kernels' own product and wait code on one CTA and leaves one product out.  Every thread has
to give up on it, and, whatever number of products is called before and after, keep the phase it gave up on: a phase
that moved on would name an earlier product, which has landed, and the tensor memory would be freed at once.
The group has to agree to leave.

Results of a device on which a wait ran out may be wrong, so every call that waits for the device and hands on a root
has to report it, until it is cleared.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = 1024


@pytest.fixture()
def lib(pkg):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg.init(0)
    lib = pkg.load()
    yield lib
    lib.b200_tma_wait_errors()


@pytest.mark.parametrize("before", [0, 1, 2])
@pytest.mark.parametrize("after", [0, 1, 2, 5])
def test_threads_give_up_on_the_same_product(pkg, lib, before, after):
    counts = np.full(3, 7, np.uint32)
    assert lib.b200_tma_wait_errors() == 0
    pkg._check(lib.b200_probe_product_wait(before, after, counts.ctypes.data))
    assert counts.tolist() == [THREADS, 0, THREADS]
    assert lib.b200_tma_wait_errors() == 1
    assert lib.b200_tma_wait_errors() == 0


def _empty(torch, n):
    return torch.zeros(n, dtype=torch.int64, device="cuda")


NB, NBE, NC = 6, 7, 5


def _commit(pkg, torch):
    root = pkg.commit_device(_empty(torch, NC << NBE), _empty(torch, pkg.tree_num_elements(1 << NBE, 4)),
                             _empty(torch, NC << NB), NB, NBE, NC, 4, _empty(torch, NC << NB))
    return 0, root


def _commit_q(pkg, torch):
    return 0, pkg.commit_q_device(_empty(torch, 3 << NBE), _empty(torch, pkg.tree_num_elements(1 << NBE, 4)),
                                  _empty(torch, 3 << NBE), NB, NBE, 1, 3, 4, _empty(torch, 3 << NBE))


def _commit_host(pkg, torch):
    return 0, pkg.commit_host(np.zeros((1 << NB, NC), np.uint64), NBE, 4)[0]


def _stream(pkg, torch):
    words = pkg.stream_commit_slot_bytes(NB, NBE, NC, 1) // 8
    return 0, pkg.stream_commit_packed(_empty(torch, words), words, np.zeros((1 << NB, 1), np.uint64), [3] * NC, NB, NBE)


def _batch(pkg, torch):
    bufs = [_empty(torch, NC << NB), _empty(torch, NC << NB), _empty(torch, NC << NBE),
            _empty(torch, pkg.tree_num_elements(1 << NBE, 4))]
    inst = pkg.BatchInstance(*[b.data_ptr() for b in bufs], NB, NBE, NC, 4)
    roots = np.ones(4, np.uint64)
    pkg._check(pkg.load().b200_commit_batch_device(ctypes.byref(inst), 1, roots.ctypes.data, None))
    return 0, roots


def _witness(pkg, torch):
    pkg.set_hash_family(2)
    trace, root = np.zeros((1 << NB, NC), np.uint64), np.ones(4, np.uint64)
    bufs, info, params = pkg.DeviceBuffers(), pkg.StarkShape(NB, NBE, NC, 4), pkg.StepsParams(trace=trace.ctypes.data)
    lib = pkg.load()
    assert lib.commit_witness(info.setup_ptr, ctypes.byref(params), 0, 0, 0, root.ctypes.data, bufs.ptr, b"") < 64
    lib.get_stream_proofs(bufs.ptr)
    return bufs.error(), root


def _custom(pkg, torch):
    pkg.set_hash_family(2)
    trace, root, bufs = np.zeros((1 << NB, NC), np.uint64), np.ones(4, np.uint64), pkg.DeviceBuffers()
    pkg.load().write_custom_commit(root.ctypes.data, 4, NB, NBE, NC, bufs.ptr, trace.ctypes.data, b"")
    return bufs.error(), root


def _serve(pkg, torch):
    lib = pkg.load()
    trace, root = np.zeros((1 << NB, NC), np.uint64), np.zeros(4, np.uint64)
    srv = lib.b200_server_new(0, 1 << 24, 1)
    assert srv
    try:
        rid = lib.b200_server_submit(srv, trace.ctypes.data, NB, NBE, NC, 4, root.ctypes.data)
        assert rid > 0
        pkg._check(lib.b200_server_wait_all(srv, 20000))
        rc = lib.b200_server_status(srv, rid, None)
        return (0 if rc == 1 else rc), root
    finally:
        lib.b200_server_free(srv)


@pytest.mark.parametrize("call", [_commit, _commit_q, _commit_host, _stream, _batch, _witness, _custom, _serve])
def test_callers_are_told(pkg, lib, call):
    torch = pytest.importorskip("torch")

    def code():
        try:
            rc, root = call(pkg, torch)
        except pkg.B200Error as e:
            return e.code
        if rc:
            assert not np.any(root)
        else:
            assert np.any(root)
        return rc

    assert code() == 0
    pkg._check(lib.b200_probe_product_wait(0, 0, np.zeros(3, np.uint32).ctypes.data))
    assert code() == pkg.B200_ECUDA
    assert code() == pkg.B200_ECUDA
    assert lib.b200_tma_wait_errors() == 1
    assert code() == 0
