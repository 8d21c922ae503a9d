"""What the host code allocates, waits for and gives back, and what it does when an allocation fails, against a CUDA
runtime without a GPU.

A workspace that could not grow must not count as grown: the next, smaller call allocates again instead of
launching a kernel on a null pointer."""
import ctypes as C

import pytest

import host_runtime
from cupythia_b200 import _lib

OK, NOMEM = _lib.CP_OK, _lib.CP_ERR_NOMEM
NONE = 1 << 62


@pytest.fixture(scope="module")
def rt(tmp_path_factory):
    return host_runtime.load(host_runtime.build(str(tmp_path_factory.mktemp("host"))))


@pytest.fixture
def h(rt):
    rt.fake_fail_above(NONE)
    rt.fake_fail_nth(-1)
    cfg, p = _lib.cp_config(), C.c_void_p()
    assert rt.cp_config_default(C.byref(cfg)) == OK
    assert rt.cp_create(C.byref(cfg), C.byref(p)) == OK
    yield p
    rt.fake_fail_above(NONE)
    rt.fake_fail_nth(-1)
    assert rt.cp_destroy(p) == OK
    assert rt.fake_device_allocations() == 0 and rt.fake_pinned_allocations() <= 1


def _iterate(rt, h, n):
    return rt.cp_vegas_iteration(h, n, 0, 1.5, C.byref(_lib.cp_result()))


def test_flow_buffer_after_a_failed_growth(rt, h):
    assert rt.cp_flow_init(h, 7) == OK and rt.cp_flow_enable(h, 1) == OK
    assert _iterate(rt, h, 1 << 20) == OK
    rt.fake_fail_above(1 << 30)
    assert _iterate(rt, h, 1 << 28) == NOMEM
    rt.fake_watch(b"k_flow_fwd_tc", 9)
    assert _iterate(rt, h, 1 << 18) == OK
    assert rt.fake_is_device(rt.fake_watched(), 16 << 18)


def test_slots_after_a_failed_growth(rt, h):
    assert rt.cp_set_wmax(h, 1.0) == OK
    r = _lib.cp_unweight_result()
    assert rt.cp_unweight(h, 300, 0, None, 0, C.byref(r)) == OK
    rt.fake_fail_nth(0)
    assert _iterate(rt, h, 1 << 20) == NOMEM
    rt.fake_watch(b"k_unw_finish", 0)
    assert rt.cp_unweight(h, 300, 0, None, 0, C.byref(r)) == OK
    assert rt.fake_is_device(rt.fake_watched(), 64)


@pytest.mark.parametrize("nth", range(8))
def test_kinematics_after_a_failed_growth(rt, h, nth):
    def set2kin(n):
        return rt.cp_set2kin_batch(h, *[(C.c_float * n)() for _ in range(4)], n)

    assert set2kin(100) == OK
    rt.fake_fail_nth(nth)
    assert set2kin(1000) == NOMEM
    rt.fake_clear()
    assert rt.cp_sigma_hat_batch(h, 111, 21, 21, (C.c_float * 1000)()) == OK   # no batch is set
    assert rt.fake_count(b"launch") == 0
    assert set2kin(50) == OK
    assert rt.fake_count(b"malloc 200") == 8


@pytest.mark.parametrize("nth", range(5))
def test_flow_set_up_after_a_failed_allocation(rt, h, nth):
    """Every array of the flow is there once a call on the flow succeeds."""
    before = rt.fake_device_allocations()
    rt.fake_fail_nth(nth)
    assert rt.cp_flow_init(h, 7) == NOMEM
    rt.fake_watch(b"k_flow_pack", 1)
    assert rt.cp_flow_init(h, 7) == OK
    assert rt.fake_is_device(rt.fake_watched(), 64)
    assert rt.fake_device_allocations() == before + 5


def test_pinned_records_after_a_failed_growth(rt, h):
    per = (_lib.cp_result * 1000)()
    rt.fake_fail_nth(0)
    assert rt.cp_integrate(h, 1000, 64, 1.5, 0, per, C.byref(_lib.cp_result())) == NOMEM
    assert rt.cp_integrate(h, 1, 64, 1.5, 0, per, C.byref(_lib.cp_result())) == OK


def test_a_handle_s_work_ends_before_its_memory_goes(rt, h):
    """The step calls return with their kernels in flight; on the default stream, too, nothing is unpinned or freed
    before they are done."""
    cfg, p = _lib.cp_config(), C.c_void_p()
    assert rt.cp_config_default(C.byref(cfg)) == OK and rt.cp_create(C.byref(cfg), C.byref(p)) == OK
    assert rt.cp_flow_init(p, 7) == OK
    rt.fake_clear()
    assert rt.cp_flow_step_moments(p, 0, 64, (C.c_double * 2)()) == OK
    last = rt.fake_count(b"")
    assert rt.fake_first(b"sync") == -1
    assert rt.cp_destroy(p) == OK
    gone = [rt.fake_first(e) for e in (b"unpin", b"free")]
    assert last <= rt.fake_first(b"sync") < min(gone)


def test_handles_one_after_another_map_no_pinned_chunk(rt):
    """The driver maps a chunk for the first pinned allocation of a process and unmaps it with the last, which takes
    longer than all else in a handle's life: handles that come and go must not do so each time."""
    cfg, p = _lib.cp_config(), C.c_void_p()
    assert rt.cp_config_default(C.byref(cfg)) == OK
    assert rt.cp_create(C.byref(cfg), C.byref(p)) == OK and rt.cp_destroy(p) == OK
    rt.fake_clear()
    for _ in range(3):
        assert rt.cp_create(C.byref(cfg), C.byref(p)) == OK
        assert rt.cp_integrate(p, 20, 64, 1.5, 0, (_lib.cp_result * 20)(), C.byref(_lib.cp_result())) == OK
        assert rt.cp_destroy(p) == OK
    assert rt.fake_count(b"chunk") == 0
    assert rt.fake_device_allocations() == 0 and rt.fake_pinned_allocations() == 1


@pytest.mark.parametrize("nth", range(8))
def test_a_handle_that_cannot_be_made_leaves_nothing(rt, h, nth):
    cfg, p = _lib.cp_config(), C.c_void_p()
    assert rt.cp_config_default(C.byref(cfg)) == OK
    dev, pin = rt.fake_device_allocations(), rt.fake_pinned_allocations()
    rt.fake_fail_nth(nth)
    rc = rt.cp_create(C.byref(cfg), C.byref(p))
    rt.fake_fail_nth(-1)
    if rc == OK:
        assert rt.cp_destroy(p) == OK
    else:
        assert rc == NOMEM and not p.value
    assert (rt.fake_device_allocations(), rt.fake_pinned_allocations()) == (dev, pin)


@pytest.mark.parametrize("produce", ["unweight", "generate_host"])
def test_production_gives_the_training_buffers_back(rt, h, produce):
    """Training keeps its buffers for the next call and over a few production passes; the eighth in a row frees
    them, but not those of a step that is not finished."""
    n, chunk = 300, (C.c_uint8 * (300 * 64 + 16))()
    at = (C.addressof(chunk) + 15) & ~15

    def pass_():
        r = _lib.cp_unweight_result()
        if produce == "unweight":
            return rt.cp_unweight(h, n, 0, at, n, C.byref(r))
        return rt.cp_generate_host(h, n, 0, n, at, n, C.byref(r))

    assert rt.cp_set_wmax(h, 1.0) == OK and rt.cp_flow_init(h, 7) == OK
    assert pass_() == OK and rt.cp_flow_sample(h, 0, 64, 0, 0, at) == OK
    before = rt.fake_device_bytes()
    assert rt.cp_flow_train(h, 1, 4096, 1e-3, None) == OK
    kept = rt.fake_device_bytes() - before
    assert 2000 * 4096 < kept < 1 << 30
    for _ in range(2):
        assert all(pass_() == OK for _ in range(7))
        assert rt.fake_device_bytes() == before + kept
        assert rt.cp_flow_train(h, 1, 4096, 1e-3, None) == OK
    assert all(pass_() == OK for _ in range(8))
    assert rt.fake_device_bytes() == before
    moments, loss = (C.c_double * 2)(), C.c_double()
    assert rt.cp_flow_step_moments(h, 0, 4096, moments) == OK
    assert all(pass_() == OK for _ in range(9))
    assert rt.fake_device_bytes() == before + kept
    assert rt.cp_flow_step_gradient(h, moments, 4096, None, C.byref(loss)) == OK
