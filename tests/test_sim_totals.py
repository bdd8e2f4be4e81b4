"""DeviceSim.conservation's call, without a GPU (the library call is a fake):
every call has a result of its own, also where two threads sum one state at the
same time, and takes the arrays as they are then."""
import ctypes
import threading


class FakeTensor:
    def __init__(self, ptr):
        self.ptr = ptr

    def data_ptr(self):
        return self.ptr


def make_sim(fake):
    from flow_gb300.sim import DeviceSim
    sim = DeviceSim.__new__(DeviceSim)
    sim.nx, sim.ny = 12, 10
    sim.a = {"rho": FakeTensor(4096), "e": FakeTensor(8192), "reduce": FakeTensor(12288)}
    sim._conservation = fake
    return sim


def address(p):
    if isinstance(p, int):
        return p
    return ctypes.cast(p, ctypes.c_void_p).value


def write_pair(out, a, b):
    pair = (ctypes.c_double * 2).from_address(address(out))
    pair[0], pair[1] = a, b


def test_two_threads_have_results_of_their_own():
    both_wrote = threading.Barrier(2, timeout=30)
    got = {}

    def fake(nx, ny, pad, rho, e, reduce, out, sync):
        n = float(threading.current_thread().name)
        write_pair(out, n, 10.0 * n)
        both_wrote.wait()
        return 0

    sim = make_sim(fake)

    def call():
        got[threading.current_thread().name] = sim.conservation()

    threads = [threading.Thread(target=call, name=str(n)) for n in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == {"1": (1.0, 10.0), "2": (2.0, 20.0)}


def test_takes_the_arrays_of_the_call():
    seen = []

    def fake(nx, ny, pad, rho, e, reduce, out, sync):
        seen.append((nx, ny, pad, address(rho), address(e), address(reduce), sync))
        write_pair(out, 3.0, 4.0)
        return 0

    sim = make_sim(fake)
    assert sim.conservation() == (3.0, 4.0)
    sim.a["rho"] = FakeTensor(65536)
    assert sim.conservation() == (3.0, 4.0)
    assert seen == [(12, 10, 2, 4096, 8192, 12288, 1), (12, 10, 2, 65536, 8192, 12288, 1)]
