"""Device inputs and results of one value set (symgb_set_arg_sets_device,
symgb_get_result_sets_device): the copy kernel's 16-byte and 8-byte paths, odd
starts and lengths and several blocks, and the runtime's copies that stand in
for it (a pointer that is no multiple of 8).  Exact mode, bit for bit, from a
first run launch by launch to replayed ones with other inputs."""
import ctypes as C

import numpy as np
import pytest

from symboliclib_gb300 import native

import oracle.cpu as ocpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 8, 4])
@pytest.mark.parametrize("kind", [native.SCHEDULE_PLAIN, native.SCHEDULE_LEVELS])
@pytest.mark.parametrize("name,size", [("cloth", 3), ("cotan", 27), ("ata", 9)])
def test_inputs_and_results_at_any_address(name, size, kind, offset):
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload(name, size, 7)
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=kind, math=native.MATH_EXACT)
    n = u.output_length[0]
    rng = np.random.default_rng(size + offset)
    for _ in range(4):
        inputs = [a * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for a in w.inputs]
        ref = ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, inputs)[0]
        buffers = []
        for a in inputs:
            b = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
            b[offset:offset + a.nbytes] = torch.from_numpy(a.view(np.uint8)).cuda()
            buffers.append(b)
        out = torch.full((n * 8 + 16,), 0x5a, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for i, b in enumerate(buffers):
            native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(b.data_ptr() + offset), i))
        native.check(lib.symgb_run_async(u.handle))
        native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(out.data_ptr() + offset), 0))
        native.check(lib.symgb_synchronize(u.handle))
        got = out.cpu().numpy()
        assert np.array_equal(got[offset:offset + n * 8], ref.view(np.uint8))
        assert np.all(got[:offset] == 0x5a) and np.all(got[offset + n * 8:] == 0x5a)


def test_page_locked_memory_of_the_host():
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload("cotan", 8, 7)
    ref = ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, w.inputs)[0]
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=native.SCHEDULE_LEVELS, math=native.MATH_EXACT)
    a = torch.from_numpy(w.inputs[0].copy()).pin_memory()
    out = torch.empty(len(ref), dtype=torch.float64).pin_memory()
    native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(a.data_ptr()), 0))
    native.check(lib.symgb_run_async(u.handle))
    native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(out.data_ptr()), 0))
    native.check(lib.symgb_synchronize(u.handle))
    assert np.array_equal(out.numpy().view(np.uint64), ref.view(np.uint64))


@pytest.mark.parametrize("sets", [1, 3, 9])
def test_inputs_made_on_another_stream(sets):
    """The unit's stream waits for an event behind which another stream writes
    the inputs, late; the copy launched after that wait, though chained to what
    precedes it, takes the new values."""
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload("cotan", 8, 7)
    rng = np.random.default_rng(sets)
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=native.SCHEDULE_LEVELS, math=native.MATH_EXACT)
    u.set_num_sets(sets)
    other, own = torch.cuda.Stream(), torch.cuda.Stream()
    native.check(lib.symgb_set_stream(u.handle, C.c_void_p(own.cuda_stream)))
    a = torch.zeros(u.arg_length[0] * sets, dtype=torch.float64, device="cuda")
    out = torch.zeros(u.output_length[0] * sets, dtype=torch.float64, device="cuda")
    for _ in range(8):
        ins = [w.inputs[0] * (1 + 1e-3 * rng.uniform(-1, 1, a.numel() // sets)) for _ in range(sets)]
        ref = np.concatenate([ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, [i])[0] for i in ins])
        new = torch.from_numpy(np.concatenate(ins)).cuda()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            torch.cuda._sleep(1000000)  # half a millisecond
            a.copy_(new)
            done = other.record_event()
        with torch.cuda.stream(own):
            out.zero_()
            own.wait_event(done)
        native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(a.data_ptr()), 0))
        native.check(lib.symgb_run_async(u.handle))
        native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(out.data_ptr()), 0))
        native.check(lib.symgb_synchronize(u.handle))
        assert np.array_equal(out.cpu().numpy().view(np.uint64), ref.view(np.uint64))
