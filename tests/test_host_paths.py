"""Host paths of libdgfock that decide which quartets a call evaluates, and
what it does when a CUDA call fails, on a CUDA runtime without a GPU
(fake_cudart.cpp, preloaded in a child process): kernels do not run, their
launches are checked against the live allocations and the quartets that they
cover are counted."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = """
import ctypes, json, os, sys
sys.path.insert(0, {root!r})
import numpy as np
from dalton_b200 import _lib, molecules
from dalton_b200.basis import build_basis
from dalton_b200.fock import FockBuilder

F = ctypes.CDLL({fake!r})
F.fake_kernels.restype = F.fake_bad.restype = ctypes.c_char_p
for n in ("fake_quartets", "fake_not_once", "fake_launches", "fake_replays", "fake_streams", "fake_live", "fake_malloc_calls"):
    getattr(F, n).restype = ctypes.c_long
F.fake_fail_malloc.argtypes = [ctypes.c_long] * 2

def builder(basis, n=1):
    return FockBuilder(build_basis(molecules.water_cluster(n, seed=2), basis))

def status(f, *a, **k):
    try:
        f(*a, **k)
    except _lib.DgfError as e:
        return e.status
    return 0

def covered(f=None):
    if f is not None:
        F.fake_reset()
        f()
    return dict(quartets=F.fake_quartets(), not_once=F.fake_not_once(), bad=F.fake_bad().decode(),
                kernels=F.fake_kernels().decode().split())

def eye(fb):
    return np.eye(fb.nbf)

def out(**kw):
    print("RESULT " + json.dumps(kw))
"""


@pytest.fixture(scope="session")
def host(tmp_path_factory):
    """Runs a snippet in a child with the fake runtime; returns its result."""
    lib = str(tmp_path_factory.mktemp("fake") / "libfakecudart.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "dalton_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", lib], check=True)

    def run(code):
        src = PRELUDE.format(root=ROOT, fake=lib) + textwrap.dedent(code)
        r = subprocess.run([sys.executable, "-c", src], env=dict(os.environ, LD_PRELOAD=lib), capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads([ln for ln in r.stdout.splitlines() if ln.startswith("RESULT ")][-1][7:])

    return run


SHARDS = """
basis, n = {basis!r}, 3
whole = covered(lambda: builder(basis).herfck(eye(builder(basis)), thrs=1e-6))
fbs = [builder(basis) for _ in range(n)]
{setup}
F.fake_reset()
got = [status(fb.herfck, eye(fb), thrs=1e-6, shard=(r, n)) for r, fb in enumerate(fbs)]
out(whole=whole, got=got, parts=covered())
"""


@pytest.mark.parametrize("basis", ["cc-pVDZ", "6-31G*", "STO-3G", "cc-pVTZ"])
@pytest.mark.parametrize("state", ["alike", "pinned", "copied", "stored"])
def test_shards_tile_whatever_a_rank_did_before(host, basis, state):
    """The shards of one build cover every quartet once, also where one
    rank's context was pinned to other kernels, took over such a tuning, or
    holds an integral store: none of these may move its cut points."""
    setup = {"alike": "", "pinned": "fbs[0].set_class_kernel((1, 0, 0, 0), 0)",
             "copied": "p = builder(basis); p.set_class_kernel((1, 0, 1, 0), 0); fbs[0].copy_tuning_from(p)",
             "stored": "_lib.check(_lib.load().dgf_store_integrals(fbs[0]._h, 1e-6, 0, None, None), 'store')"}[state]
    r = host(SHARDS.format(basis=basis, setup=setup))
    assert r["got"] == [0, 0, 0]
    assert r["parts"]["quartets"] == r["whole"]["quartets"] and r["parts"]["not_once"] == 0
    assert r["parts"]["bad"] == ""


@pytest.mark.parametrize("basis", ["6-31G*", "cc-pVTZ"])
def test_shard_without_memory_is_an_error(host, basis):
    """A rank that cannot allocate what the others' shards use (the resolved
    context of a segmented basis, the pair fragments of the pack kernels)
    reports it instead of cutting the queue another way, and builds its shard
    once there is memory; a whole build goes on with what it has.  One
    allocation of a first build fails, or a run of them."""
    r = host(f"""
    basis, n = {basis!r}, 2
    other = builder(basis)
    d = eye(other)
    whole = covered(lambda: other.herfck(d, thrs=1e-6))
    fb = builder(basis)
    calls = F.fake_malloc_calls()
    fb.herfck(d, thrs=1e-6, shard=(0, n))
    calls = F.fake_malloc_calls() - calls
    sharded, alone = [], []
    for k, fails in [(k, m) for k in range(calls) for m in (1, 6)]:
        for shard, res in ((n, sharded), (1, alone)):
            fb = builder(basis)
            F.fake_reset()
            F.fake_fail_malloc(k, fails)
            s = status(fb.herfck, d, thrs=1e-6, shard=(0, shard))
            F.fake_fail_malloc(0, 0)
            why = _lib.last_error() if s else ''
            if s:
                F.fake_reset()
                assert status(fb.herfck, d, thrs=1e-6, shard=(0, shard)) == 0
            if shard > 1:
                other.herfck(d, thrs=1e-6, shard=(1, n))
            c = covered()
            res.append([s, c["quartets"] - whole["quartets"], c["not_once"], c["bad"], why])
    out(sharded=sharded, alone=alone)
    """)
    if basis == "6-31G*":
        assert any(s[0] and not a[0] for s, a in zip(r["sharded"], r["alone"]))
    assert any("pair fragments" in s[4] for s in r["sharded"])
    assert not any("pair fragments" in a[4] for a in r["alone"])
    for s, missing, not_once, bad, _ in r["sharded"]:
        assert s in (0, 2, 3) and (missing, not_once, bad) == (0, 0, ""), r["sharded"]
    for s, missing, not_once, bad, _ in r["alone"]:
        assert s in (0, 2, 3) and (not_once, bad) == (0, ""), r["alone"]


@pytest.mark.parametrize("basis", ["cc-pVDZ", "cc-pVTZ", "6-31G*"])
def test_failed_plan_does_not_stay(host, basis):
    """A build whose plan for another threshold could not be made leaves
    nothing behind that a later build would read: each allocation of the
    second threshold's build fails once, then the first threshold's build and
    the second's are made again."""
    r = host(f"""
    basis = {basis!r}
    a, b = 1e-2, 1e-7
    ref = builder(basis)
    d = eye(ref)
    whole = [covered(lambda: ref.herfck(d, thrs=t)) for t in (a, b)]
    fb = builder(basis)
    fb.herfck(d, thrs=a)
    calls = F.fake_malloc_calls()
    fb.herfck(d, thrs=b)
    calls = F.fake_malloc_calls() - calls
    res = []
    for k in range(calls):
        fb = builder(basis)
        for _ in range(3):
            fb.herfck(d, thrs=a)
        F.fake_fail_malloc(k, 1)
        s = status(fb.herfck, d, thrs=b)
        F.fake_fail_malloc(0, 0)
        for t, w in zip((a, a, b), (whole[0], whole[0], whole[1])):
            c = covered(lambda: fb.herfck(d, thrs=t))
            res.append([k, s, c["quartets"] - w["quartets"], c["not_once"], c["bad"]])
    out(res=res)
    """)
    assert any(s for _, s, *_ in r["res"])
    for k, s, missing, not_once, bad in r["res"]:
        assert (missing, not_once, bad) == (0, 0, ""), (k, s, missing, not_once, bad)


def test_failed_batch_plan_does_not_stay(host):
    """The same for a batch, whose graph refers to the plan's buffers."""
    r = host("""
    from dalton_b200.batch import BatchBuilder
    fbs = [builder("cc-pVDZ", n) for n in (1, 2)]
    bb = BatchBuilder(fbs)
    buf = np.zeros(2 * bb.total)

    def build(t):
        opt = _lib.default_options(thrs=t)
        p = buf.ctypes.data
        return _lib.load().dgf_fock_batch(bb._h, p, p + 8 * bb.total, ctypes.byref(opt), 1, None, None)

    a, b = 1e-2, 1e-7
    F.fake_reset()
    assert build(a) == 0
    n = F.fake_quartets()
    calls = F.fake_malloc_calls()
    assert build(b) == 0
    calls = F.fake_malloc_calls() - calls
    res = []
    for k in range(calls):
        assert build(a) == 0
        F.fake_fail_malloc(k, 1)
        s = build(b)
        F.fake_fail_malloc(0, 0)
        for _ in range(2):
            F.fake_reset()
            r = build(a)
            res.append([s, r, F.fake_quartets() - n, F.fake_not_once(), F.fake_bad().decode()])
    out(res=res)
    """)
    assert len(r["res"]) >= 6 and all(x == [2, 0, 0, 0, ""] for x in r["res"]), r["res"]


@pytest.mark.parametrize("basis", ["6-31G*", "cc-pVDZ"])
def test_capture_after_a_store(host, basis):
    """Inside the caller's stream capture, where nothing can be allocated, a
    direct build runs on the plan that a store made, as every context does
    whose own direct builds use that plan; a shard, which must not, says what
    it needs."""
    r = host(f"""
    fb, other = builder({basis!r}), builder({basis!r})
    lib = _lib.load()
    t = 1e-6
    assert lib.dgf_store_integrals(fb._h, t, 0, None, None) == 0
    buf = np.zeros((2, fb.nbf, fb.nbf))
    ift = (_lib.dgf_int * 1)(13)

    def build(b, n=1, **o):
        opt = _lib.default_options(thrs=t, shard_count=n, **o)
        F.fake_reset()
        s = lib.dgf_fock_device(b._h, 1, ift, buf[0].ctypes.data, buf[1].ctypes.data, ctypes.byref(opt), None, None)
        return [s, F.fake_quartets(), F.fake_not_once(), F.fake_bad().decode()]

    F.fake_user_capture(1)
    captured, shard, screened = build(fb), build(fb, 2), build(fb, ifthrs=10)
    F.fake_user_capture(0)
    other.set_class_kernel((1, 0, 0, 0), 0)  # serves its whole builds itself
    own = build(other)
    after = [build(fb), build(fb, 2)]
    F.fake_user_capture(1)
    again = [build(fb), build(fb, 2)]
    out(captured=captured, shard=shard, screened=screened, own=own, after=after, again=again)
    """)
    assert r["captured"] == r["own"] and r["own"][0] == 0 and r["own"][3] == ""
    assert r["shard"][0] == (1 if basis == "6-31G*" else 0)
    assert r["screened"][0] != 0  # its buffers were not there: an error, not a crash
    assert [x[0] for x in r["after"] + r["again"]] == [0] * 4
    assert r["after"] == r["again"]


def test_build_without_a_graph(host):
    """A short build whose graph cannot be made is launched without one, and
    replayed as a graph once it can be."""
    r = host("""
    fb = builder("cc-pVDZ")
    d = eye(fb)
    F.fake_fail_instantiate(2)
    res = []
    for _ in range(8):
        replays = F.fake_replays()
        F.fake_reset()
        s = status(fb.herfck, d, thrs=1e-6)
        res.append([s, F.fake_quartets(), F.fake_not_once(), F.fake_bad().decode(), F.fake_replays() - replays,
                    fb.last_stats["kernel_launches"]])
    out(res=res)
    """)
    assert r["res"][0][1] > 0
    for x in r["res"]:
        assert x[:4] == [0, r["res"][0][1], 0, ""] and x[5] == r["res"][0][5], r["res"]
    assert [x[4] for x in r["res"]] == [0, 0, 0, 0, 0, 1, 1, 1]


@pytest.mark.parametrize("basis", ["cc-pVDZ", "6-31G*", "cc-pVTZ"])
def test_launches_wait_for_uploads(host, basis):
    """No kernel runs on one of the library's own streams, which do not wait
    for the legacy stream, while a cudaMemcpy may still be on its way to the
    device; and no plan is replaced while a build on another stream may still
    read it."""
    r = host(f"""
    from dalton_b200.batch import BatchBuilder
    F.fake_reset()
    fb = builder({basis!r})
    res = dict(create=F.fake_bad().decode())
    for name, call in dict(
            count=lambda: fb.ao_quartets(1e-6), fock=lambda: fb.herfck(eye(fb), thrs=1e-6),
            screened=lambda: fb.herfck(eye(fb), thrs=1e-6, ifthrs=10), one=lambda: fb.oneint(),
            grad=lambda: fb.grad2e(eye(fb)) if {basis!r} != "cc-pVTZ" else None).items():
        F.fake_reset()
        call()
        res[name] = F.fake_bad().decode()
    lib, ift, stream = _lib.load(), (_lib.dgf_int * 1)(13), np.zeros(1)
    buf = np.zeros((2, fb.nbf, fb.nbf))
    F.fake_reset()
    for t in (1e-6, 1e-2, 1e-6, 1e-4):  # asynchronous builds on the caller's stream, one plan after the other
        opt = _lib.default_options(thrs=t)
        assert lib.dgf_fock_device(fb._h, 1, ift, buf[0].ctypes.data, buf[1].ctypes.data, ctypes.byref(opt),
                                   stream.ctypes.data, None) == 0
    res["plans"] = F.fake_bad().decode()
    F.fake_reset()
    bb = BatchBuilder([fb, builder({basis!r}, 2)])
    p = np.zeros(2 * bb.total)
    for t in (1e-4, 1e-2, 1e-4):
        opt = _lib.default_options(thrs=t)
        assert lib.dgf_fock_batch(bb._h, p.ctypes.data, p.ctypes.data + 8 * bb.total, ctypes.byref(opt), 0,
                                  stream.ctypes.data, None) == 0
    res["batch"] = F.fake_bad().decode()
    out(**res)
    """)
    assert r == {k: "" for k in r}


@pytest.mark.parametrize("basis", ["cc-pVDZ", "6-31G*"])
def test_contexts_of_a_batch_stay_small(host, basis):
    """A context makes its launch streams and tables with its first plan: one
    that only takes part in batches holds its own stream and no more, nor does
    its resolved form."""
    r = host(f"""
    from dalton_b200.batch import BatchBuilder
    fbs = [builder({basis!r}, n) for n in (1, 2, 1)]
    made = F.fake_streams()
    bb = BatchBuilder(fbs)
    batch = F.fake_streams() - made
    live = F.fake_live()
    F.fake_reset()
    fbs[0].herfck(eye(fbs[0]), thrs=1e-6)
    first = F.fake_streams() - made - batch
    fbs[0].herfck(eye(fbs[0]), thrs=1e-4)
    fbs[0].grad2e(eye(fbs[0]))
    later = F.fake_streams() - made - batch - first
    bb.close()
    for fb in fbs:
        fb.close()
    out(made=made, batch=batch, first=first, later=later, left=[F.fake_streams(), F.fake_live()], bad=F.fake_bad().decode())
    """)
    forms = 2 if basis == "6-31G*" else 1
    assert r["made"] == 3
    assert r["batch"] == 5 + 3 * (forms - 1)  # its own five, and one of each resolved form
    assert (r["first"], r["later"]) == (7, 0)
    assert r["left"] == [0, 0] and r["bad"] == ""


# 10 X + Y per density; a general one (X = 0) takes two of the eight slots that
# are built at once
MANY = [[13] * 8, [13] * 9, [3] * 5, [13, 3, 3, 3, 3], [22, 2, 1, 11, 23, 3], [13] * 7 + [3, 3, 13], [13] * 15 + [3] * 8]


@pytest.mark.parametrize("ifctyp", MANY)
def test_many_densities_stay_in_their_buffers(host, ifctyp):
    """More density slots than are built at once: every combination of half
    Fock matrices lies in their buffer."""
    r = host(f"""
    fb = builder("cc-pVDZ")
    ict = {ifctyp!r}
    d = np.zeros((len(ict), fb.nbf, fb.nbf))
    F.fake_reset()
    s = status(fb.herfck, d, ict, thrs=1e-4)
    out(s=s, bad=F.fake_bad().decode())
    """)
    assert r == dict(s=0, bad="")
