"""The work that users of the commit path have it do, as cases for timing and comparison.

A case is one call (or the call and its harvest) of the public entry points on inputs that are
ready where the caller has them: device buffers for the native API, host memory for the calls that
take a host trace.  Every output is a whole number (field elements as canonical 64-bit words,
digests, roots), so two correct implementations agree bit for bit.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The framework's package (its folder's name has a hyphen, so it is loaded by path)."""
    name = "pil2_proofman_b200"
    if name not in sys.modules:
        path = os.path.join(os.getcwd(), "pil2-proofman_b200", "__init__.py")
        if not os.path.exists(path):
            path = os.path.join(REPO, "pil2-proofman_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path, submodule_search_locations=[os.path.dirname(path)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # the smallest AIRs of a proof (range checks, short tables): launches and latency count
        dict(name="commit_tiny", kind="commit", nbits=9, blowup=1, ncols=19, arity=4, family=2, rowmajor=True),
        # the 2^16 x 32 single commit of the benchmark
        dict(name="commit_small", kind="commit", nbits=16, blowup=1, ncols=32, arity=4, family=2, rowmajor=True),
        # an ordinary AIR with an odd width, its trace already column-major (as a previous stage leaves it)
        dict(name="commit_ragged", kind="commit", nbits=18, blowup=1, ncols=101, arity=4, family=2, rowmajor=False),
        # the benchmark's default workload: one large AIR, 2^22 x 256, blowup 2
        dict(name="commit_large", kind="commit", nbits=22, blowup=1, ncols=256, arity=4, family=2, rowmajor=True),
        # stage-2-style commit with the extension columns as limbs, 780 words a row, blowup 4
        dict(name="commit_stage2", kind="commit", nbits=19, blowup=2, ncols=780, arity=4, family=2, rowmajor=True),
        # final compression stage: binary tree (width-8 sponge), high blowup
        dict(name="commit_final", kind="commit", nbits=16, blowup=4, ncols=54, arity=2, family=2, rowmajor=True),
        # the other hash family (Poseidon1), same path
        dict(name="commit_poseidon1", kind="commit", nbits=18, blowup=1, ncols=64, arity=4, family=1, rowmajor=True),
        # many instances of uneven size committed as one batch
        dict(name="batch_mixed", kind="batch", count=24, lo=10, hi=17, maxcols=128, shapes_seed=7),
        # quotient stage: 3-limb quotient, two chunks, committed with its tree
        dict(name="q_stage", kind="q", nbits=20, blowup=1, qdeg=2, qdim=3, arity=4),
        # bit-packed host rows committed through a streaming slot (no full LDE is kept)
        dict(name="stream_packed", kind="stream", nbits=18, blowup=1, ncols=53, width=23, family=2),
        # the reference's own call: a host trace through commit_witness to its root, from pinned memory
        dict(name="witness_host", kind="witness", nbits=18, blowup=1, ncols=180),
        # FRI query openings read from a resident commit
        dict(name="openings", kind="openings", nbits=18, blowup=1, ncols=120, arity=4, queries=228),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# LDE words of the largest listed commit: a drawn one stays below
_MAX_LDE = (1 << 23) * 256


def draw(rng):
    kind = rng.choice(["commit", "commit", "commit", "commit", "batch", "q", "stream", "witness", "openings"])
    if kind == "commit":
        blowup = rng.choice([1, 1, 1, 2, 2, 3, 4])
        nbits = rng.randint(8, 22 - blowup)
        cap = max(2, min(780, _MAX_LDE >> (nbits + blowup + 1)))
        # Poseidon1 and the narrow sponges cost up to twice a column's time
        arity = rng.choice([4, 4, 4, 3, 2])
        return dict(kind=kind, nbits=nbits, blowup=blowup, ncols=_logint(rng, 2, cap), arity=arity,
                    family=rng.choice([2, 2, 2, 1]), rowmajor=rng.random() < 0.7)
    if kind == "batch":
        lo = rng.randint(8, 12)
        return dict(kind=kind, count=rng.randint(4, 31), lo=lo, hi=lo + rng.randint(2, 6),
                    maxcols=_logint(rng, 24, 200), shapes_seed=rng.randrange(1 << 20))
    if kind == "q":
        blowup = rng.choice([1, 2, 3])
        return dict(kind=kind, nbits=rng.randint(9, 21 - blowup), blowup=blowup, qdeg=rng.randint(1, 1 << blowup),
                    qdim=3, arity=rng.choice([4, 4, 3, 2]))
    if kind == "stream":
        return dict(kind=kind, nbits=rng.randint(10, 19), blowup=rng.choice([1, 1, 2]), ncols=rng.randint(2, 64),
                    width=rng.randint(1, 60), family=rng.choice([1, 2]))
    if kind == "witness":
        nbits = rng.randint(9, 19)
        return dict(kind=kind, nbits=nbits, blowup=rng.choice([1, 1, 2]), ncols=_logint(rng, 3, 250))
    return dict(kind=kind, nbits=rng.randint(10, 19), blowup=rng.choice([1, 1, 2]), ncols=_logint(rng, 4, 400),
                arity=rng.choice([4, 4, 3, 2]), queries=_logint(rng, 16, 1024))


def _batch_shapes(case):
    """(nbits, nbits_ext, ncols) of a batch's instances: log2 rows and widths uniform, a quarter at blowup 4."""
    r = np.random.RandomState(case["shapes_seed"])
    out = []
    for i in range(case["count"]):
        nbits = int(r.randint(case["lo"], case["hi"] + 1))
        out.append((nbits, nbits + (2 if i % 4 == 3 else 1), int(r.randint(8, case["maxcols"] + 1))))
    return out


class _Plan:
    """A batched plan and the buffers it points to."""

    def __init__(self, pkg, shapes, traces):
        self.pkg, self.lib, self.traces = pkg, pkg.load(), traces
        self.ldes, self.trees, self.scratch = [], [], []
        arr = (pkg.BatchInstance * len(shapes))()
        for i, (nbits, nbits_ext, ncols) in enumerate(shapes):
            self.scratch.append(_empty(pkg.lde_scratch_words(nbits, ncols)))
            self.ldes.append(_empty(ncols, 1 << nbits_ext))
            self.trees.append(_empty(pkg.tree_num_elements(1 << nbits_ext, 4)))
            arr[i] = pkg.BatchInstance(traces[i].data_ptr(), self.scratch[i].data_ptr(), self.ldes[i].data_ptr(),
                                       self.trees[i].data_ptr(), nbits, nbits_ext, ncols, 4)
        self.roots = np.zeros((len(shapes), 4), dtype=np.uint64)
        self.ptr = self.lib.b200_batch_plan_new(ctypes.cast(arr, ctypes.c_void_p), len(shapes))
        if not self.ptr:
            raise RuntimeError((self.lib.b200_last_error() or b"").decode())

    def run(self):
        self.pkg._check(self.lib.b200_batch_plan_run(self.ptr, self.roots.ctypes.data, None, 0))

    def __del__(self):
        if getattr(self, "ptr", None):
            self.lib.b200_batch_plan_free(self.ptr)


class _Witness:
    """A prover's device buffers, its setup and a pinned host trace."""

    def __init__(self, pkg, case, seed):
        nbits = case["nbits"]
        self.pkg = pkg
        self.trace = torch.from_numpy(_host_random(pkg, (1 << nbits) * case["ncols"], seed)).pin_memory()
        self.bufs = pkg.DeviceBuffers()
        self.info = pkg.StarkShape(nbits, nbits + case["blowup"], case["ncols"], 4)
        self.root = np.zeros(4, dtype=np.uint64)
        self.params = pkg.StepsParams(trace=self.trace.data_ptr())


def _empty(*shape):
    return torch.empty(shape, dtype=torch.int64, device="cuda")


def _random(pkg, seed, *shape):
    """Uniform field elements on the device."""
    t = _empty(*shape)
    pkg.fill_random_device(t, t.numel(), seed)
    return t


def _host_random(pkg, n, seed):
    return pkg.fill_random_host(n, seed).view(np.int64)


def prepare(case, seed):
    pkg = _package()
    pkg.init(0)
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        traces = [_random(pkg, seed * 1000 + i, 1 << nbits, ncols) for i, (nbits, _, ncols) in enumerate(shapes)]
        torch.cuda.synchronize()
        return dict(case=case, pkg=pkg, plan=_Plan(pkg, shapes, traces))
    nbits, nbits_ext = case["nbits"], case["nbits"] + case["blowup"]
    n, next_ = 1 << nbits, 1 << nbits_ext
    if kind == "witness":
        pkg.set_hash_family(2)
        return dict(case=case, pkg=pkg, w=_Witness(pkg, case, seed))
    s = dict(case=case, pkg=pkg)
    if kind == "stream":
        rng = np.random.RandomState(seed % (1 << 31))
        widths = [int(w) for w in 1 + rng.randint(0, case["width"], case["ncols"])]
        wpr = pkg.packed_words_per_row(widths)
        packed = _host_random(pkg, n * wpr, seed).reshape(n, wpr)
        s.update(widths=widths, packed=packed.view(np.uint64), words=pkg.stream_commit_slot_bytes(
            nbits, nbits_ext, case["ncols"], wpr) // 8)
        s["slot"] = _empty(s["words"])
        return s
    s["tree"] = _empty(pkg.tree_num_elements(next_, case["arity"]))
    if kind == "q":
        s["q"] = _random(pkg, seed, next_, case["qdim"])
        s["cmq"] = _empty(case["qdeg"] * case["qdim"], next_)
        s["scratch"] = _empty(pkg.q_scratch_words(nbits_ext, case["qdim"]))
        return s
    ncols = case["ncols"]
    if kind == "openings":
        # a resident commit: openings read any LDE and tree words, so random ones serve as well
        s["lde"] = _random(pkg, seed, ncols, next_)
        pkg.fill_random_device(s["tree"], s["tree"].numel(), seed + 1)
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["rows"] = torch.randint(0, next_, (case["queries"],), generator=g, dtype=torch.int64, device="cuda")
        s["out"] = _empty(case["queries"], pkg.query_proof_words(next_, ncols, case["arity"], 0))
        return s
    s["trace"] = _random(pkg, seed, *((n, ncols) if case["rowmajor"] else (ncols, n)))
    s["scratch"] = _empty(pkg.lde_scratch_words(nbits, ncols))
    s["lde"] = _empty(ncols, next_)
    return s


def run(state):
    case, pkg = state["case"], state["pkg"]
    kind = case["kind"]
    if kind == "batch":
        plan = state["plan"]
        plan.run()
        return dict(roots=plan.roots.view(np.int64), ldes=plan.ldes, trees=plan.trees)
    nbits, nbits_ext = case["nbits"], case["nbits"] + case["blowup"]
    if kind == "commit":
        if pkg.native_hash_family() != case["family"]:
            pkg.set_native_hash_family(case["family"])
        root = pkg.commit_device(state["lde"], state["tree"], state["trace"], nbits, nbits_ext, case["ncols"],
                                 case["arity"], state["scratch"], trace_rowmajor=case["rowmajor"])
        if case["family"] != 2:
            pkg.set_native_hash_family(2)
        return dict(root=root.view(np.int64), lde=state["lde"], tree=state["tree"])
    if kind == "q":
        root = pkg.commit_q_device(state["cmq"], state["tree"], state["q"], nbits, nbits_ext, case["qdeg"],
                                   case["qdim"], case["arity"], state["scratch"])
        return dict(root=root.view(np.int64), cmq=state["cmq"], tree=state["tree"])
    if kind == "stream":
        if pkg.native_hash_family() != case["family"]:
            pkg.set_native_hash_family(case["family"])
        root = pkg.stream_commit_packed(state["slot"], state["words"], state["packed"], state["widths"], nbits,
                                        nbits_ext)
        if case["family"] != 2:
            pkg.set_native_hash_family(2)
        return dict(root=root.view(np.int64))
    if kind == "witness":
        w, lib = state["w"], pkg.load()
        slot = lib.commit_witness(w.info.setup_ptr, ctypes.byref(w.params), 0, 0, 0, w.root.ctypes.data, w.bufs.ptr, b"")
        if slot == 2**64 - 1:
            raise RuntimeError((lib.b200_last_error() or b"").decode())
        lib.get_stream_proofs(w.bufs.ptr)
        return dict(root=w.root.view(np.int64))
    pkg.query_openings_device(state["out"], state["lde"], 1 << nbits_ext, case["ncols"], state["tree"], case["arity"],
                              state["rows"], case["queries"])
    return dict(openings=state["out"])


# field multiplications of one permutation (S-boxes of the 8 full and 22 partial rounds, and the
# linear layers' full-word products)
_MULS = {2: {w: 8 * w * 4 + 22 * (4 + w) for w in (8, 12, 16)},
         1: {w: 8 * w * 4 + w * w + 22 * (4 + w + w - 1) for w in (8, 12, 16)}}


def _tree_work(rows, ncols, arity, family):
    """(bytes written, field multiplications) of a tree over `rows` rows of `ncols` words."""
    w = 4 * arity
    perms = rows * -(-ncols // (w - 4))
    nodes, level = rows, rows
    while level > 1:
        level = -(-level // arity)
        perms += level
        nodes += level
    return nodes * 32, perms * _MULS[family][w]


def _lde_work(nbits, nbits_ext, ncols):
    """(bytes, field multiplications) of one extension: trace in, LDE out, one product per butterfly."""
    n, next_ = 1 << nbits, 1 << nbits_ext
    return 8 * ncols * (n + next_), ncols * (n // 2 + next_ // 2) * nbits


def work(case):
    """Bytes: inputs read once and outputs written once.  flops: two per field multiplication."""
    kind = case["kind"]
    if kind == "batch":
        b = m = 0
        for nbits, nbits_ext, ncols in _batch_shapes(case):
            lb, lm = _lde_work(nbits, nbits_ext, ncols)
            tb, tm = _tree_work(1 << nbits_ext, ncols, 4, 2)
            b, m = b + lb + tb, m + lm + tm
        return dict(bytes=b, flops=2 * m)
    nbits, nbits_ext = case["nbits"], case["nbits"] + case["blowup"]
    n, next_ = 1 << nbits, 1 << nbits_ext
    if kind == "openings":
        levels = math.ceil(round(nbits_ext / math.log2(case["arity"]), 9))
        words = case["queries"] * (case["ncols"] + levels * (case["arity"] - 1) * 4)
        return dict(bytes=16 * words, flops=0)
    if kind == "q":
        cols = case["qdeg"] * case["qdim"]
        tb, tm = _tree_work(next_, cols, case["arity"], 2)
        muls = case["qdim"] * (next_ // 2) * nbits_ext + cols * (next_ // 2) * nbits
        return dict(bytes=8 * next_ * (case["qdim"] + cols) + tb, flops=2 * (muls + tm))
    lb, lm = _lde_work(nbits, nbits_ext, case["ncols"])
    tb, tm = _tree_work(next_, case["ncols"], case.get("arity", 4), case.get("family", 2))
    if kind == "stream":  # packed rows in (about half the drawn width a column), the tree out
        return dict(bytes=n * case["ncols"] * case["width"] // 16 + tb, flops=2 * (lm + tm))
    return dict(bytes=lb + tb, flops=2 * (lm + tm))


def tolerance(case):
    """Field elements and digests are canonical integers: every correct implementation gives these bits."""
    return "exact"
