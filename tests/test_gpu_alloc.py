"""The library's device memory: buffers given back while another thread captures a
graph, the surplus of the pool, its memory for a large buffer when the device is full,
objects made, used and dropped by several threads at once, and the handle of a state's m."""
import ctypes as C
import threading

import numpy as np
import pytest

from helpers import random_m

M = pytest.importorskip("magnumaf")
torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _stepped(shape, seed=1, stream=None):
    """An integrator (its work buffer: 8 x 24 bytes per cell) after one DP45 step, and its state."""
    st = M.State(M.Mesh(*shape, 3e-9, 3e-9, 3e-9), 8e5, random_m(shape, seed))
    llg = M.LLGIntegrator(0.1, [M.ExchangeField(1.3e-11)], "DP45", hmax=1e-14)
    llg.step(st)
    return llg, st


def _capture_while(meanwhile):
    """A graph captured in thread-local mode while another thread runs `meanwhile`, and replayed."""
    x = torch.ones(1000, device="cuda")
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    raised = []

    def run():
        try:
            meanwhile()
        except M.MafError as e:
            raised.append(e)

    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        y = x + 1
        t = threading.Thread(target=run)
        t.start()
        t.join()
        y = 2 * y
    assert not raised
    g.replay()
    torch.cuda.synchronize()
    assert torch.all(y == 4)
    return g, y


def test_buffers_dropped_while_another_thread_captures():
    graphs = [_capture_while(lambda: None)]  # what the first capture of a process allocates is not counted
    made = [_stepped((512, 512, 2)) for _ in range(6)]  # 100 MB of pool memory each
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    graphs.append(_capture_while(made.clear))
    _stepped((8, 8, 1))  # an object made and dropped afterwards gives back what was pending
    M.trim_memory()
    # all of the 6 x 126 MB came back (but for torch's graph memory)
    assert torch.cuda.mem_get_info()[0] - free0 >= (6 * 126 - 64) * MB


@pytest.mark.parametrize("prec", ["fp64", "fp32_field"])
@pytest.mark.parametrize("shape", [(64, 64, 1), (100, 25, 1)])
def test_first_evaluation_while_another_thread_captures(shape, prec):
    """A new mesh's tensor, tables and FP32 copies are made without waiting for the whole device."""
    mesh, m = M.Mesh(*shape, 3e-9, 3e-9, 3e-9), random_m(shape, 4)
    want = M.DemagField(mesh).H_in_Apm(M.State(mesh, 8e5, m, precision=prec))
    got = []
    _capture_while(lambda: got.append(M.DemagField(mesh).H_in_Apm(M.State(mesh, 8e5, m, precision=prec))))
    assert np.array_equal(got[0], want)


def test_pool_gives_its_memory_to_a_large_buffer():
    """With 200 MB left on the device and as much unused in the pool, a 300 MB state is made."""
    made = [_stepped((512, 512, 2)) for _ in range(2)]
    del made
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 200 * MB, dtype=torch.uint8, device="cuda")
    try:
        m = np.zeros((300, 200, 205, 3), order="F")
        m[..., 2] = 1.0
        st = M.State(M.Mesh(300, 200, 205, 1e-9, 1e-9, 1e-9), 8e5, m)
        assert tuple(st.mean_m()) == (0.0, 0.0, 1.0)
        with pytest.raises(M.MafError) as e:  # and what does not fit is still an error
            M.State(M.Mesh(600, 200, 205, 1e-9, 1e-9, 1e-9), 8e5, np.concatenate([m, m]))
        assert e.value.code == 3
        del st
    finally:
        del fill
        torch.cuda.empty_cache()
    _stepped((64, 64, 1))


def test_threads_make_use_and_drop_objects():
    shapes = [(64, 48, 1), (33, 20, 3), (100, 25, 1), (300, 100, 2)]  # tensors on kernels of 1 to 64 KB

    def run(shape, seed):
        st = M.State(M.Mesh(*shape, 3e-9, 3e-9, 3e-9), 8e5, random_m(shape, seed))
        llg = M.LLGIntegrator(0.1, [M.DemagField(st.mesh), M.ExchangeField(1.3e-11)], "RKF45", hmax=1e-14)
        llg.steps(st, 5)
        return np.asarray(st.m).copy()

    want = {(i, k): run(s, k) for i, s in enumerate(shapes) for k in range(3)}
    bad = []

    def worker(i):
        for rep in range(30):
            for k in range(3):
                try:
                    if not np.array_equal(run(shapes[i], k), want[i, k]):
                        bad.append((i, k, rep))
                except M.MafError as e:
                    bad.append((i, k, rep, str(e)))

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(len(shapes)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("shape", [(8, 6, 1), (300, 200, 3)])
def test_device_m_has_an_ipc_handle(shape):
    """State.device_m points to an allocation of its own (cudaMalloc), before and after steps."""
    rt = C.CDLL("libcudart.so.12")  # torch's; the context is shared
    st = M.State(M.Mesh(*shape, 3e-9, 3e-9, 3e-9), 8e5, random_m(shape, 2))
    terms = [M.ExchangeField(1.3e-11)]
    llg = M.LLGIntegrator(0.1, terms, "RKF45", hmax=1e-14)
    it = M.Stochastic_LLG(0.1, 300.0, 1e-14, st, terms, "Heun", seed=1)
    for use in (lambda: None, lambda: llg.step(st), lambda: it.step(st), lambda: llg.steps(st, 2)):
        use()
        st.mean_m()  # waits for the state's stream
        handle = (C.c_char * 64)()
        assert rt.cudaIpcGetMemHandle(handle, C.c_void_p(st.device_m())) == 0


def test_many_integrators_keep_their_own_error_norm():
    """More integrators at once than one page of pinned words holds (512), some dropped and
    made anew in between: each reads its own norm."""
    st = M.State(M.Mesh(6, 5, 1, 3e-9, 3e-9, 3e-9), 8e5, random_m((6, 5, 1), 3))
    term = M.ExchangeField(1.3e-11)

    def make(i):
        return M.LLGIntegrator(0.1, [term], "RKF45", atol=1e-6 * (i + 1))

    def norm(llg):
        return llg.rk_attempt(st, "RKF45", 2e-14)[1]

    want = [norm(make(i)) for i in range(1100)]  # one after the other
    assert len(set(want)) == len(want)
    made = [make(i) for i in range(1100)]
    assert [norm(llg) for llg in made] == want
    for i in list(range(0, 1100, 3)) + list(range(512, 1024)):
        made[i] = None
    for i in range(1100):
        if made[i] is None:
            made[i] = make(i)
            assert norm(made[i]) == want[i]
    assert [norm(llg) for llg in made] == want


def test_unused_buffers_are_kept_within_bounds_and_given_back():
    """States dropped and made again reuse their m buffers; what is kept unused stays below 512
    MB, trim_memory gives it back, and a state made of a used buffer holds its own m."""
    shape = (512, 512, 2)
    _stepped(shape)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    M.trim_memory()
    free0 = torch.cuda.mem_get_info()[0]
    made = [_stepped(shape, seed) for seed in range(14)]  # 96 MB of the pool and twice 12 of m each
    assert free0 - torch.cuda.mem_get_info()[0] >= 14 * (96 + 2 * 12) * MB
    made.clear()
    big = [M.State(M.Mesh(512, 512, 16, 1e-9, 1e-9, 1e-9), 8e5, np.ones((512, 512, 16, 3)))
           for _ in range(4)]  # 4 x 101 MB of m
    big.clear()
    assert free0 - torch.cuda.mem_get_info()[0] < 512 * MB + 32 * MB
    m = random_m(shape, 77)
    st = M.State(M.Mesh(*shape, 3e-9, 3e-9, 3e-9), 8e5, m)
    np.testing.assert_allclose(np.asarray(st.m), m, rtol=0, atol=1e-15)
    del st
    M.trim_memory()
    assert free0 - torch.cuda.mem_get_info()[0] < 16 * MB
