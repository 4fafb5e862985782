"""Runs of six or more launches are replayed as graphs from their second time
on: every run takes its own inputs, whatever was changed since the graph was
made, in a capture of the caller's and beside one.  Exact mode, bit for bit."""
import ctypes as C
import threading

import numpy as np
import pytest

from symboliclib_gb300 import native

import oracle.cpu as ocpu

pytestmark = pytest.mark.gpu

EXECUTORS = [native.EXEC_COMPILED, native.EXEC_INTERPRETER]


def drawn(w, rng, sets=1):
    """Inputs of `sets` value sets and the results the oracle gives for them."""
    ins = [[a * (1 + 1e-3 * rng.uniform(-1, 1, a.size)) for _ in range(sets)] for a in w.inputs]
    ref = [ocpu.evaluate(w.plan, w.index_data, w.out_index_data, w.const_data, [a[s] for a in ins])[0]
           for s in range(sets)]
    return [np.concatenate(a) for a in ins], np.concatenate(ref)


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def plain_unit(w, executor):
    u = native.Unit.from_workload(w)
    u.set_schedule(kind=native.SCHEDULE_PLAIN, math=native.MATH_EXACT, executor=executor)
    return u


@pytest.mark.parametrize("executor", EXECUTORS)
def test_every_run_follows_inputs_and_configuration(executor):
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload("cotan", 8, 3)
    rng = np.random.default_rng(1)
    u = plain_unit(w, executor)
    stream = torch.cuda.Stream()
    changes = [lambda: None,
               lambda: native.check(lib.symgb_set_stream(u.handle, C.c_void_p(stream.cuda_stream))),
               lambda: u.set_num_sets(3), lambda: u.set_num_sets(1),
               lambda: native.check(lib.symgb_set_stream(u.handle, None)),
               lambda: u.set_direct_outputs(False), lambda: u.set_direct_outputs(True),
               lambda: u.set_kernel_shape(0, 2, 0, 64), lambda: u.set_load_path(native.LOAD_L2),
               lambda: u.set_item_layout(native.ITEMS_GROUPED),
               lambda: u.set_schedule(kind=native.SCHEDULE_PLAIN, math=native.MATH_EXACT, executor=executor, use_graph=1)]
    for n, change in enumerate(changes):
        change()
        for run in range(3):
            ins, ref = drawn(w, rng, u.num_sets)
            for i, a in enumerate(ins):
                u.set_arg(i, a)
            u.run()
            assert u.last_launch_count() == w.plan.contents.num_kernels
            assert same(u.get_result(0), ref), (n, run)


@pytest.mark.parametrize("executor", EXECUTORS)
def test_runs_in_a_capture_of_the_callers(executor):
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload("cotan", 8, 3)
    rng = np.random.default_rng(2)
    u = plain_unit(w, executor)
    stream = torch.cuda.Stream()
    native.check(lib.symgb_set_stream(u.handle, C.c_void_p(stream.cuda_stream)))
    a = torch.zeros(u.arg_length[0], dtype=torch.float64, device="cuda")
    out = torch.zeros(u.output_length[0], dtype=torch.float64, device="cuda")

    def enqueue():
        native.check(lib.symgb_set_arg_sets_device(u.handle, C.c_void_p(a.data_ptr()), 0))
        native.check(lib.symgb_run_async(u.handle))
        native.check(lib.symgb_get_result_sets_device(u.handle, C.c_void_p(out.data_ptr()), 0))

    def check(go):
        ins, ref = drawn(w, rng)
        a.copy_(torch.from_numpy(ins[0]))
        torch.cuda.synchronize()
        go()
        torch.cuda.synchronize()
        assert same(out.cpu().numpy(), ref)
    for _ in range(3):  # launch by launch, then replayed
        check(enqueue)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        enqueue()
    for _ in range(3):
        check(graph.replay)
    check(enqueue)


@pytest.mark.parametrize("executor", EXECUTORS)
@pytest.mark.parametrize("same_thread", [False, True])
def test_a_graph_made_beside_a_capture_of_the_callers(executor, same_thread):
    """The second run makes its graph while another stream is being captured in
    the mode that forbids everyone what could disturb it."""
    torch = pytest.importorskip("torch")
    lib = native.symgb()
    w = native.Workload("cotan", 8, 3)
    ins, ref = drawn(w, np.random.default_rng(3))
    u = plain_unit(w, executor)
    u.set_arg(0, ins[0])
    u.run()
    t = torch.ones(100, device="cuda")
    torch.cuda.synchronize()
    codes = []

    def work():
        codes.extend([lib.symgb_run_async(u.handle), lib.symgb_run_async(u.handle)])
        codes.append(lib.symgb_set_barrier_limits(u.handle, 10 ** 9, 0))  # drops the graph
        codes.append(lib.symgb_run_async(u.handle))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        double = t * 2
        if same_thread:
            work()
        else:
            thread = threading.Thread(target=work)
            thread.start()
            thread.join()
        four = double * 2
    assert codes == [0, 0, 0, 0], native.symgb().symgb_last_error()
    graph.replay()
    torch.cuda.synchronize()
    assert bool((four == 4).all())
    assert same(u.get_result(0), ref)
