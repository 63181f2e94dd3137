"""The library's host code on a CUDA runtime of host memory (fake_runtime.cpp), in place of a GPU: what a
captured run may be used for again, what a failed allocation leaves behind, and what the memory that the
library keeps does to later calls.  The kernels do nothing but keep an epoch's counts (every agent cites
itself), so results of the sampling are not looked at here."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import paragraph_gb300 as pg
from paragraph_gb300 import PG_ERR_CAPACITY, PG_ERR_STATE, PG_WEIGHTS_REFCOMPAT, GrowthEngine, PAParams, PGError, RCParams, TraceInput
from paragraph_gb300.build import PKG, ROOT, build_library, nvcc


def build_fake(d):
    """The library on the fake runtime, built in directory d."""
    cuda = Path(nvcc()).resolve().parents[1] / "include"
    if not list((PKG / "_build").glob("*.o")):
        build_library(force=True)
    objs = sorted(str(p) for p in (PKG / "_build").glob("*.o"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-I", str(cuda), "-I", str(ROOT / "include"), "-o", str(d / "libfake.so"),
                    str(ROOT / "tests" / "fake_runtime.cpp"), *objs, "-lpthread"], check=True)
    lib = pg.load_library(d / "libfake.so")
    lib.fake_reset.argtypes = [C.c_int64, C.c_int32]
    lib.fake_fail_in.argtypes = [C.c_int64]
    lib.fake_hold.argtypes = lib.fake_ball.argtypes = [C.c_int64]
    for f in ("fake_mallocs", "fake_faults", "fake_pool_idle", "fake_memory_queries", "fake_free_bytes", "fake_hold"):
        getattr(lib, f).restype = C.c_int64
    lib.fake_launches.argtypes = [C.c_char_p]
    lib.fake_launches.restype = C.c_int32
    lib.fake_dependent_range.argtypes = [C.c_char_p, C.POINTER(C.c_int64), C.POINTER(C.c_int64)]
    lib.fake_page_locked.argtypes = [C.c_int64]
    lib.fake_page_locked.restype = C.c_void_p
    lib.fake_page_locked_free.argtypes = [C.c_void_p]
    return lib


@pytest.fixture(scope="module")
def fake(built, tmp_path_factory):
    return build_fake(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def host(fake, monkeypatch):
    """Engines made in the test run on the fake runtime."""
    monkeypatch.setattr(pg, "_lib", fake)
    fake.fake_reset(64 << 30, 152)
    return fake


def _engine(n=1000, new=40, epochs=8, **kw):
    eng = GrowthEngine(seed=1, **kw)
    eng.load_graph(np.zeros(n, np.int32), np.ones(n, np.float32), np.zeros(0, np.int32), np.zeros(0, np.int32),
                   PAParams(fixed_new_nodes=new, growth_rate=0.0), planned_epochs=epochs)
    return eng


class _PageLocked:
    def __init__(self, lib, count):
        self.lib, self.p = lib, lib.fake_page_locked(4 * count)
        self.a = np.ctypeslib.as_array((C.c_int32 * count).from_address(self.p))
        self.a[:] = -7

    def free(self):
        self.a = None
        self.lib.fake_page_locked_free(self.p)


# ---------------------------------------------------------------- captured runs
def test_captured_run_follows_its_output_buffers(host):
    """A run repeated from a checkpoint with the same page-locked sources and other targets writes the
    targets it was given."""
    bufs = [_PageLocked(host, 1000) for _ in range(3)]
    src, d1, d2 = (b.a for b in bufs)
    with _engine() as eng:
        eng.checkpoint()
        ne, counts = eng.run_epochs_out(3, (src, d1))
        assert ne == 120 and (d1[:120] == np.arange(1000, 1120)).all() and counts.sum() == 120
        d1[:] = -7
        eng.restore()
        ne, _ = eng.run_epochs_out(3, (src, d2))
        assert ne == 120 and (d2[:120] == np.arange(1000, 1120)).all()
        assert (d1 == -7).all()
    del src, d1, d2
    for b in bufs:
        b.free()


@pytest.mark.parametrize("page_locked", [False, True])
def test_captured_run_follows_its_capacity(host, page_locked):
    """Buffers of another length from the same checkpoint: too short is reported and nothing is written past
    the end, long enough again is no error."""
    bufs = [_PageLocked(host, 1000) for _ in range(2)] if page_locked else []
    s, d = (b.a for b in bufs) if page_locked else (np.full(1000, -7, np.int32), np.full(1000, -7, np.int32))
    with _engine() as eng:
        eng.checkpoint()
        for cap in (120, 100, 1000, 40, 39, 120):
            s[:], d[:] = -7, -7
            if cap >= 120:
                assert eng.run_epochs_out(3, (s[:cap], d[:cap]))[0] == 120
                done = 120
            else:
                with pytest.raises(PGError) as err:
                    eng.run_epochs_out(3, (s[:cap], d[:cap]))
                assert err.value.status == PG_ERR_CAPACITY
                done = cap // 40 * 40
            for a in (s, d):
                assert (a[:done] == np.arange(1000, 1000 + done)).all() and (a[done:] == -7).all()
            eng.restore()
    del s, d
    for b in bufs:
        b.free()


def test_captured_run_follows_the_graph_it_starts_from(host):
    """The same epoch number reached with another number of nodes: the captured run was for other epochs'
    agents."""
    with _engine(epochs=12) as eng:
        eng.set_params(PAParams(growth_rate=0.05, fixed_new_nodes=0))
        eng.reserve(6000, 6000)
        eng.checkpoint()
        eng.run_er_epochs(3, 10, 1e-3)
        first = eng.run_epochs(2)
        eng.restore()
        eng.run_er_epochs(3, 400, 1e-3)
        n0 = eng.counts()[0]
        again = eng.run_epochs(2)
        assert again == eng.counts()[0] - n0 > first


def test_captured_run_is_used_again(host):
    """Nothing changed: the run is not captured a second time."""
    with _engine() as eng:
        eng.checkpoint()
        out = (np.empty(500, np.int32), np.empty(500, np.int32))
        eng.run_epochs_out(3, out)
        eng.restore()
        host.fake_clear_launches()
        eng.run_epochs_out(3, out)
        assert host.fake_launches(b"k_epoch_begin") == 0


# ---------------------------------------------------------------- checkpoints
def test_failed_checkpoint_leaves_nothing_to_restore(host):
    """A second checkpoint that fails on the way has overwritten parts of the first: a restore is refused,
    and the next whole checkpoint is restored."""
    with _engine() as eng:
        eng.checkpoint()  # no citations yet: one copied range fewer than later
        eng.run_epochs(2)
        host.fake_fail_in(0)
        with pytest.raises(PGError):
            eng.checkpoint()
        with pytest.raises(PGError) as err:
            eng.restore()
        assert err.value.status == PG_ERR_STATE
        assert host.fake_faults() == 0
        host.fake_fail_in(-1)
        eng.checkpoint()
        at = eng.counts()
        eng.run_epochs(1)
        eng.restore()
        assert eng.counts() == at == (1080, 80)


def test_refused_checkpoint_keeps_the_earlier_one(host):
    with GrowthEngine(seed=1) as eng:
        with pytest.raises(PGError):
            eng.checkpoint()
    with _engine() as eng:
        eng.checkpoint()
        eng.run_epochs(1)
        eng.restore()
        assert eng.counts() == (1000, 0)


# ---------------------------------------------------------------- failed loads
@pytest.mark.parametrize("weight_model", [0, PG_WEIGHTS_REFCOMPAT])
def test_load_after_a_failed_load(host, weight_model):
    """Whichever device allocation of a load fails, the next load has everything its epochs use."""
    seed = [np.zeros(500, np.int32), np.ones(500, np.float32), np.zeros(0, np.int32), np.zeros(0, np.int32)]
    prm = PAParams(fixed_new_nodes=20, growth_rate=0.0)
    failed = 0
    for n in range(100):
        with GrowthEngine(seed=1, weight_model=weight_model) as eng:
            host.fake_fail_in(n)
            try:
                eng.load_graph(*seed, prm, planned_epochs=2)
            except PGError:
                failed += 1
            else:
                break
            finally:
                host.fake_fail_in(-1)
            eng.load_graph(*seed, prm, planned_epochs=2)
            if weight_model:
                eng.rc_configure(RCParams(growth_rate=0.04), np.full(10, 5), np.full(4, 0.25))
            assert eng.run_epochs(2) >= 40
    assert failed >= (8 if weight_model else 1) and host.fake_faults() == 0


# ---------------------------------------------------------------- the likelihood's weight table
def _trace(n, agents):
    """`agents` papers of one epoch, each with one citation, after a seed of n."""
    t = n + agents
    return TraceInput(pub=np.zeros(t, np.int32), fitness=np.ones(t, np.float32), seed_src=np.zeros(0, np.int32),
                      seed_dst=np.zeros(0, np.int32), epoch_nodes=np.array([n, t]), epoch_t=np.array([0]),
                      anchors=np.tile(np.array([0, -1, -1, -1], np.int32), (agents, 1)),
                      cite_off=np.arange(agents + 1), cites=np.zeros(agents, np.int32), num_anchors=1)


def _points(b):
    return np.tile([1.0, 5.0, 1.0, 4.0], (b, 1))


def test_refused_weight_table_is_asked_for_once(host):
    """The table of 64 points has no room (51 MB of 200 MB free, an eighth may be taken), that of 4 points has:
    batches in turn neither free and allocate nor ask for the free memory again, and the small batches keep
    their table."""
    host.fake_ball(16_000)
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(_trace(200_000, 100))
        held = host.fake_free_bytes() - (200 << 20)
        host.fake_hold(held)
        for b in (4, 64):
            eng.loglik(_points(b))
            eng.loglik_grad(_points(b))
        host.fake_clear_launches()
        before = host.fake_mallocs(), host.fake_memory_queries()
        for b in (64, 4, 64, 4):
            eng.loglik(_points(b))
            eng.loglik_grad(_points(b))
        assert (host.fake_mallocs(), host.fake_memory_queries()) == before
        assert host.fake_launches(b"k_lik_table1") == 4 and host.fake_launches(b"k_lik_eval") == 4
        host.fake_hold(-held)
        eng.load_trace(_trace(200_000, 100))  # another trace asks again
        host.fake_clear_launches()
        eng.loglik(_points(64))
        assert host.fake_launches(b"k_lik_table2") == 1


def test_larger_weight_table_counts_the_one_it_replaces(host):
    host.fake_ball(16_000)
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(_trace(200_000, 100))
        eng.loglik(_points(32))  # 26 MB
        eng.loglik(_points(64))  # the buffers of 64 points
        eng.load_trace(_trace(200_000, 100))
        eng.loglik(_points(32))
        held = host.fake_free_bytes() - (400 << 20)
        host.fake_hold(held)
        host.fake_clear_launches()
        eng.loglik(_points(64))  # 51 MB of 400 + 26
        assert host.fake_launches(b"k_lik_table2") == 1
        host.fake_hold(-held)


# ---------------------------------------------------------------- temporaries kept between calls
def _pool_idle(host, edges=3_000_000):
    """A context whose load of `edges` citations of few papers has left the temporaries' pool that much idle."""
    eng = GrowthEngine(seed=1)
    eng.load_graph(np.zeros(1000, np.int32), np.ones(1000, np.float32), np.ones(edges, np.int32),
                   np.zeros(edges, np.int32), PAParams(fixed_new_nodes=10, growth_rate=0.0), planned_epochs=1)
    assert host.fake_pool_idle() > 40 * edges
    return eng


def test_an_export_gives_its_memory_back(host):
    """Attribute rows of 6M papers take over 500 MB of temporaries, of which the load had left 144 MB reserved: at
    most 256 MB are."""
    n = 6_000_000
    with _engine(n=n) as eng:
        free, idle = host.fake_free_bytes(), host.fake_pool_idle()
        rows = dict(ids=np.arange(n), draws=np.zeros((n, 4)), ints=np.zeros((n, 4), np.int32),
                    generators=np.full((n, 4), -1, np.int64))
        for _ in range(2):
            assert _attributes(host, eng, rows) == pg.PG_OK
            assert host.fake_free_bytes() >= free - ((256 << 20) - idle)


def _attributes(host, eng, rows):
    r = pg._AttrRows()
    for k, v in rows.items():
        setattr(r, k, v.ctypes.data)
    r.num_nodes, r.num_seed = len(rows["ids"]), 0
    size = C.c_int64()
    return host.pg_format_attributes(eng._ctx, 0, C.byref(r), None, 0, C.byref(size))


def test_idle_temporaries_count_as_free(host):
    """51 MB of weight table, where an eighth of 350 MB free is too little and of 350 MB and the pool's idle
    memory enough; and the allocation finds its room in the pool's."""
    host.fake_ball(16_000)
    with _pool_idle(host, 6_000_000), GrowthEngine(seed=1) as eng:
        eng.load_trace(_trace(200_000, 100))
        held = host.fake_free_bytes() - (350 << 20)
        host.fake_hold(held)
        host.fake_clear_launches()
        eng.loglik(_points(64))
        assert host.fake_launches(b"k_lik_table2") == 1
        host.fake_hold(-held)


def test_an_allocation_takes_back_idle_temporaries(host):
    def load(eng, n=200_000):
        eng.load_graph(np.zeros(n, np.int32), np.ones(n, np.float32), np.zeros(0, np.int32), np.zeros(0, np.int32),
                       PAParams(fixed_new_nodes=10, growth_rate=0.0), planned_epochs=1)

    with _pool_idle(host), GrowthEngine(seed=1) as eng:
        with GrowthEngine(seed=1) as other:
            free = host.fake_free_bytes()
            load(other)
            arena = free - host.fake_free_bytes()
        held = host.fake_free_bytes() - (arena - (10 << 20))
        host.fake_hold(held)
        load(eng)
        assert eng.counts() == (200_000, 0)
        host.fake_hold(-held)


# ---------------------------------------------------------------- dependent launches
@pytest.mark.parametrize("sms", [152, 76, 20])
def test_dependent_launches_follow_the_device(built, tmp_path, sms):
    """Launches of more than 1,280 threads per SM of the device are plain ones, whatever its number of SMs.  The
    number is asked for once per process: a process each."""
    code = f"""
import sys, ctypes as C
sys.path[:0] = [{str(ROOT)!r}, {str(ROOT / 'tests')!r}]
import paragraph_gb300 as pg, test_host_state_cpu as t
lib = pg._lib = t.build_fake(t.Path({str(tmp_path)!r}))
lib.fake_reset(64 << 30, {sms})
for new in (10, 300, 900, 1200, 4000, 7000):
    with t._engine(new=new, epochs=1) as eng:
        eng.run_epochs(1, use_graph=False)
most, least = C.c_int64(), C.c_int64()
for k in (b"k_agent_setup", b"k_bwd_place", b"k_agents<"):
    lib.fake_dependent_range(k, C.byref(most), C.byref(least))
    print(k.decode(), most.value, least.value)
"""
    out = subprocess.run([sys.executable, "-c", code], check=True, capture_output=True, text=True).stdout
    limit = sms * 1280
    seen = [tuple(map(int, line.split()[1:])) for line in out.splitlines()]
    assert len(seen) == 3
    assert all(0 < most <= limit for most, _ in seen), out
    assert all(least == 0 or least > limit for _, least in seen), out
    if sms < 152:
        assert any(least for _, least in seen), out
