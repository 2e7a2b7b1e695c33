"""Index algebra of the FFT-pass chain's line transform (gen_fft in
maos_b200/csrc/shwfs_gen.cuh), restated on the CPU in float64 with the line
strides read from that file.

A line of N points is transformed by T = N / 16 threads of 16 points: thread t
brings x[T i + t], leaves X[t + T i], and exchanges through the slots
k (T + 1) + t of its line.  Checked: the slots of a line are distinct, end
before the next line's and are all written before they are read; every
twiddle index is inside the table; the result is numpy's transform (N times
its inverse), also when a second transform follows without a reordering; the
threads of a line are lanes of one warp where only a warp barrier separates the
exchange's two sides (row passes); and the half warps' exchanges fall on
distinct banks, in both thread layouts.  No GPU."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "maos_b200", "csrc", "shwfs_gen.cuh")
THREADS, POINTS = 128, 2048


def _strides():
    """gen_ls(n, rows) as {(n, rows): stride}."""
    with open(SRC) as f:
        m = re.search(r"return n == 64 \? \(rows \? (\d+) : (\d+)\) : n == 128 \? \(rows \? (\d+) : (\d+)\) : \(rows \? (\d+) : (\d+)\);",
                      f.read())
    v = [int(x) for x in m.groups()]
    return {(n, rows): v[2 * i + (not rows)] for i, n in enumerate((64, 128, 256)) for rows in (True, False)}


def _gen_fft(v, direction):
    """v[t, i]: the threads' registers, before and after."""
    T = v.shape[0]
    N, M = 16 * T, 16 // T
    table = np.exp(-2j * np.pi * np.arange(N) / N)
    dft = (lambda a: np.fft.fft(a, axis=-1)) if direction < 0 else (lambda a: np.fft.ifft(a, axis=-1) * a.shape[-1])
    ex = np.full(16 * (T + 1), np.nan, complex)
    for t in range(T):
        w = dft(v[t])
        for k in range(16):
            tw = table[t * k]  # an index outside the table raises
            ex[k * (T + 1) + t] = w[k] * (tw if direction < 0 else np.conj(tw))
    out = np.empty_like(v)
    for t in range(T):
        for m in range(M):
            u = dft(ex[(t + T * m) * (T + 1) + np.arange(T)])
            out[t, m + M * np.arange(T)] = u
    return out


@pytest.mark.parametrize("N", [64, 128, 256])
def test_line_transform(N):
    T = N // 16
    rng = np.random.default_rng(N)
    x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    take = lambda a: np.stack([a[T * np.arange(16) + t] for t in range(T)])  # noqa: E731
    give = lambda v: v.T.reshape(-1)  # element t + T i from v[t, i]  # noqa: E731
    f = _gen_fft(take(x), -1)
    assert np.abs(give(f) - np.fft.fft(x)).max() < 1e-11 * N
    assert np.abs(give(_gen_fft(f, 1)) - N * x).max() < 1e-11 * N * N
    g = _gen_fft(_gen_fft(take(x), 1), -1)
    assert np.abs(give(g) - N * x).max() < 1e-11 * N * N


@pytest.mark.parametrize("N", [64, 128, 256])
@pytest.mark.parametrize("rows", [True, False])
def test_exchange_slots(N, rows):
    T, L, LS = N // 16, POINTS // N, _strides()[N, rows]
    M = 16 // T
    assert THREADS == L * T
    tid = np.arange(THREADS)
    line, t = (tid // T, tid % T) if rows else (tid % L, tid // L)
    if rows:
        assert all(len(set(tid[line == k] // 32)) == 1 for k in range(L))
    put = np.stack([line * LS + k * (T + 1) + t for k in range(16)])
    get = np.stack([line * LS + (t + T * m) * (T + 1) + j for m in range(M) for j in range(T)])
    for a in (put, get):
        assert len(np.unique(a)) == a.size and a.max() < L * LS
        assert all(line[k] * LS <= a[:, k].min() and a[:, k].max() < (line[k] + 1) * LS for k in tid)
        # 8-byte accesses: the lanes of a half warp on distinct pairs of banks
        assert all(len(set(r[h:h + 16] % 16)) == 16 for r in a for h in range(0, THREADS, 16))
    assert np.array_equal(np.unique(put), np.unique(get))
