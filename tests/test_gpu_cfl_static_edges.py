"""amr_cfl_dt_static at the edges of its reduction: blocks whose speed is NaN,
infinite or only the density, cell sizes that are zero, negative or NaN, the
cap of 1e6, one block to the largest accepted number, calls in a row of
different sizes and after a NaN, and calls on two streams at once.  Expected
values from numpy in the reference's order of operations (main.cpp:209-228,
misc.cpp:71-79), bit for bit."""
import ctypes

import numpy as np
import pytest

GAMMA = 1.4


def speeds(U, ng):
    """Largest speed of each block [n, 8, e, e]; NaN where a cell's is."""
    u = U[:, :, ng:-ng, ng:-ng]
    with np.errstate(all="ignore"):
        r = u[:, 0]
        v = [u[:, k] / r for k in (1, 2, 3)]
        p = (GAMMA - 1) * (u[:, 4] - 0.5 * r * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]))
        b2 = u[:, 5] * u[:, 5] + u[:, 6] * u[:, 6] + u[:, 7] * u[:, 7]
        p = p - (GAMMA - 1) * (0.5 * b2)
        ca, a = np.sqrt(b2 / r), np.sqrt(GAMMA * p / r)
        i0, i1 = (ca * ca) + (a * a), (ca * ca) - (a * a)
        out = []
        for k in (5, 6):
            can = np.sqrt((u[:, k] * u[:, k]) / r)
            out.append(np.sqrt(0.5 * (i0 + np.sqrt(i1 * i1 + 4. * (a * a) * ((ca * ca) - (can * can))))))
        s = np.maximum(np.abs(r) + out[0], np.abs(v[0]) + out[1])   # NaN if either is
    return s.reshape(len(U), -1).max(1)


def expected(U, dxdy, ng):
    with np.errstate(all="ignore"):
        h = np.where(dxdy[:, 1] < dxdy[:, 0], dxdy[:, 1], dxdy[:, 0])   # std::min: a NaN dy is passed over
        v = h / speeds(U, ng)
    return np.nan if np.isnan(v).any() else min(1e6, v.min())


def blocks(n, ng, seed):
    g = np.random.default_rng(seed)
    e = 16 + 2 * ng
    U = g.uniform(0.1, 1.0, (n, 8, e, e))
    U[:, 1:4] -= 0.5
    U[:, 5:8] -= 0.5
    U[:, 4] = g.uniform(0.1, 2.0, (n, e, e)) + 0.5 * (U[:, 1:4] ** 2).sum(1) / U[:, 0] + 0.5 * (U[:, 5:8] ** 2).sum(1)
    return U, np.repeat(g.uniform(0.01, 0.1, (n, 1)), 2, 1)


class Call:
    def __init__(self, gpu, U, dxdy, ng, copies=1, last=None):
        import torch
        self.torch, self.lib, self.ng = torch, gpu.load(), ng
        self.U = torch.from_numpy(np.ascontiguousarray(U)).cuda().repeat(copies, 1, 1, 1)
        self.d = torch.from_numpy(np.ascontiguousarray(dxdy)).cuda().repeat(copies, 1)
        self.n = len(self.U) if last is None else last
        self.out = torch.full((1,), -7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()

    def start(self, stream=None):
        stream = stream or self.torch.cuda.current_stream()
        rc = self.lib.amr_cfl_dt_static(ctypes.c_void_p(self.U.data_ptr()), self.n, self.ng,
                                        ctypes.c_void_p(self.d.data_ptr()), GAMMA,
                                        ctypes.c_void_p(self.out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))
        assert rc == 0

    def value(self):
        self.torch.cuda.synchronize()
        return self.out.item()

    def __call__(self):
        self.start()
        return self.value()


def same(got, want):
    assert got == want or (np.isnan(got) and np.isnan(want)), (got, want)


def edges():
    """name, change of (U, dxdy): one entry of each that the last of 9 blocks takes"""
    def at(k, v):
        return lambda U, d: U.__setitem__((-1, k, 9, 11), v)

    def size(a, b):
        return lambda U, d: d.__setitem__(-1, (a, b))

    def still(U, d):      # neither pressure nor field: the speed is the density
        U[-1, 1:] = 0.0

    def negatives(U, d):  # several below zero: the smallest wins
        d[2], d[5], d[7] = (-0.5, 1.0), (1.0, -3.0), (-0.25, -0.125)
    return [("plain", lambda U, d: None), ("nan_momentum", at(1, np.nan)), ("negative_pressure", at(4, -5.0)),
            ("negative_density", at(0, -0.5)), ("infinite_energy", at(4, np.inf)), ("huge_momentum", at(1, 1e200)),
            ("infinite_momentum", at(1, np.inf)), ("tiny_density", at(0, 1e-310)), ("still", still),
            ("zero_dx", size(0.0, 1.0)), ("nan_dx", size(np.nan, 1.0)), ("nan_dy", size(0.001, np.nan)),
            ("infinite_dx", size(np.inf, np.inf)), ("negatives", negatives),
            ("capped", lambda U, d: d.__setitem__(slice(None), 1e9))]


@pytest.mark.gpu
@pytest.mark.parametrize("ng", [2, 4])
@pytest.mark.parametrize("name", [e[0] for e in edges()])
def test_edge_values(gpu, name, ng):
    U, d = blocks(9, ng, 3)
    dict(edges())[name](U, d)
    call = Call(gpu, U, d, ng)
    same(call(), expected(U, d, ng))
    V, e = blocks(2, ng, 4)       # and a call after it
    same(Call(gpu, V, e, ng)(), expected(V, e, ng))


@pytest.mark.gpu
def test_calls_of_different_sizes_in_a_row(gpu):
    U, d = blocks(64, 2, 5)
    big = Call(gpu, U, d, 2, copies=1024)             # 65536 blocks, the most it takes
    big.d[-1] = 1e-4
    last = 1e-4 / speeds(U, 2)[-1]
    V, e = blocks(3, 2, 6)
    bad, f = blocks(5, 2, 7)
    bad[4, 4, 8, 8] = np.nan
    small, one, broken = Call(gpu, V, e, 2), Call(gpu, V, e, 2, last=1), Call(gpu, bad, f, 2)
    mid = Call(gpu, U, d, 2)
    for _ in range(3):
        same(small(), expected(V, e, 2))
        same(big(), min(expected(U, d, 2), last))
        same(mid(), expected(U, d, 2))
        same(broken(), np.nan)
        same(one(), expected(V[:1], e[:1], 2))


@pytest.mark.gpu
def test_calls_on_two_streams_at_once(gpu):
    """Each has its own result, and a call on one stream later is right too."""
    import torch
    U, d = blocks(64, 2, 8)
    V, e = blocks(7, 2, 9)
    a, b = Call(gpu, U, d, 2, copies=256), Call(gpu, V, e, 2)
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(10):
        a.start(sa)
        for _ in range(20):
            b.start(sb)
    same(a.value(), expected(U, d, 2))
    same(b.value(), expected(V, e, 2))
    a.out.fill_(-7.0)
    same(a(), expected(U, d, 2))


@pytest.mark.gpu
def test_captured_call(gpu):
    import torch
    U, d = blocks(40, 4, 10)
    call = Call(gpu, U, d, 4)
    call()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        call.start(s)
    for k in range(3):
        call.d[k] = 1e-3 / (k + 1)
        call.out.fill_(-7.0)
        torch.cuda.synchronize()
        g.replay()
        d[k] = 1e-3 / (k + 1)
        same(call.value(), expected(U, d, 4))
