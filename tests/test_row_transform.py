"""The row transform's index arithmetic (csrc/fft.cuh, radix_plan.h) restated in numpy and
checked on the CPU for every size, precision and row split the library builds: shared
positions stay inside each CTA's array and are a thread's own within a pass, the storage order
is a permutation, and the forward and inverse passes, run with the kernels' indices and the
tables' order, match numpy.fft. On the GPU a solve's bits are the same however its rows are split,
which served pools (whose split follows what they hold) rely on."""
import numpy as np
import pytest

from mm_propagation_b200 import capi, workloads as W

PLANS = {  # radix_plan(log2 N): log2 of the radices
    6: [1] * 6, 7: [2, 2, 2, 1], 8: [3, 3, 2], 9: [3, 3, 3], 10: [3, 3, 2, 2], 11: [3, 3, 3, 2], 12: [3, 3, 3, 3],
    13: [4, 3, 3, 3], 14: [4, 4, 4, 2], 15: [4, 4, 4, 3], 16: [4, 4, 4, 4],
}


def max_split(fp64, L):
    return 0 if L < 11 else 2 if L == 11 else 3 if L <= 13 else (16 - L if fp64 else 3 if L == 14 else 17 - L)


class Geo:
    def __init__(self, fp64, L, xc):
        r = self.r = PLANS[L]
        self.L, self.N, self.A = L, 1 << L, 1 << r[0]
        self.B, self.RM = self.N // self.A, 1 << r[-1]
        self.C = 1 << (max(0, L + (4 if fp64 else 3) - 17) + xc)
        self.RPC, self.TPR, self.NTHR = self.A // self.C, self.B // self.A, self.B // self.C
        slots = self.slots = 8 if fp64 else 16
        rs0 = self.pad(self.B)
        self.RS = rs0 + ((self.TPR - rs0) % slots if self.TPR < slots else 0)
        assert sum(r) == L and self.RPC >= 1 and self.TPR >= 1 and 32 <= self.NTHR <= (512 if fp64 else 1024)
        assert self.RPC * self.RS * (16 if fp64 else 8) <= 220 * 1024

    def pad(self, x):
        return x + x // self.slots

    def freq0(self, b):  # without k1
        k, pos, low = 0 * b, 0, self.L - self.r[0] - self.r[-1]
        for R in self.r[1:-1]:
            low -= R
            k, pos = k + (((b >> low) & ((1 << R) - 1)) << pos), pos + R
        return k << self.r[0]


def spec_pos(r, L, k):
    k1, rest, b = k & ((1 << r[0]) - 1), k >> r[0], 0 * k
    for R in r[1:-1]:
        b, rest = (b << R) | (rest & ((1 << R) - 1)), rest >> R
    return (k1 << (L - r[0])) + (rest << (L - r[0] - r[-1])) + b


def dft(v, inv):  # over the last axis, unnormalised
    return np.fft.ifft(v) * v.shape[-1] if inv else np.fft.fft(v)


def passes(g):
    """Row passes but the last: for every thread and butterfly its shared positions [r], j and L."""
    tid = np.arange(g.NTHR)
    row, u, length = tid // g.TPR, tid % g.TPR, g.B
    for p in range(1, len(g.r) - 1):
        R = 1 << g.r[p]
        S = length // R
        idx, tw = [], []
        for bf in range(g.A // R):
            b = u + g.TPR * bf
            j = b % S
            idx.append((row * g.RS + g.pad((b // S) * length + j))[:, None] + g.pad(np.arange(R) * S))
            tw.append(np.exp(-2j * np.pi * np.outer(j, np.arange(R)) / length))
        yield np.concatenate(idx), np.concatenate(tw)
        length = S
    b = np.concatenate([u + g.TPR * bf for bf in range(g.A // g.RM)])
    yield (np.tile(row, g.A // g.RM) * g.RS + g.pad(b * g.RM))[:, None] + g.pad(np.arange(g.RM)), (np.tile(row, g.A // g.RM), b)


def forward(g, x):
    s = np.full((g.C, g.RPC * g.RS), np.nan + 0j)
    for c in range(g.C):
        i = c * g.NTHR + np.arange(g.NTHR)
        v = dft(x[i[:, None] + g.B * np.arange(g.A)], False) * np.exp(-2j * np.pi * np.outer(i, np.arange(g.A)) / g.N)
        for k in range(g.A):
            s[k // g.RPC, (k % g.RPC) * g.RS + g.pad(i)] = v[:, k]
    X = np.full(g.N, np.nan + 0j)
    for c in range(g.C):
        *mid, (idx, (row, b)) = passes(g)
        for at, tw in mid:
            assert len(np.unique(at)) == at.size == g.N // g.C and at.max() < s.shape[1]
            s[c, at] = dft(s[c, at], False) * tw
        assert len(np.unique(idx)) == idx.size and idx.max() < s.shape[1]
        k1 = c * g.RPC + row
        k = (k1 + g.freq0(b))[:, None] + np.arange(g.RM) * (g.N // g.RM)
        at = (k1 * g.B + b)[:, None] + np.arange(g.RM) * (g.B // g.RM)
        assert np.array_equal(at, spec_pos(g.r, g.L, k))  # the stage kernels' order is spec_pos's
        X[at] = dft(s[c, idx], False)
    return X


def inverse(g, X):
    s = np.full((g.C, g.RPC * g.RS), np.nan + 0j)
    for c in range(g.C):
        *mid, (idx, (row, b)) = passes(g)
        at = ((c * g.RPC + row) * g.B + b)[:, None] + np.arange(g.RM) * (g.B // g.RM)
        s[c, idx] = dft(X[at], True)
        for at, tw in reversed(mid):
            s[c, at] = dft(s[c, at] * tw.conj(), True)
    x = np.full(g.N, np.nan + 0j)
    for c in range(g.C):
        i = c * g.NTHR + np.arange(g.NTHR)
        v = np.stack([s[k // g.RPC, (k % g.RPC) * g.RS + g.pad(i)] for k in range(g.A)], axis=1)
        v = v * np.exp(2j * np.pi * np.outer(i, np.arange(g.A)) / g.N)
        x[i[:, None] + g.B * np.arange(g.A)] = dft(v, True)
    return x


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("L", range(6, 17))
def test_row_transform_indices(fp64, L):
    rng = np.random.default_rng(L)
    x = rng.standard_normal(1 << L) + 1j * rng.standard_normal(1 << L)
    ref = np.fft.fft(x)
    for xc in range(max_split(fp64, L) + 1):
        g = Geo(fp64, L, xc)
        pos = spec_pos(g.r, L, np.arange(g.N))
        assert np.array_equal(np.sort(pos), np.arange(g.N))
        X = forward(g, x)
        assert np.abs(X[pos] - ref).max() < 1e-12 * np.abs(ref).max()
        y = inverse(g, X)
        assert np.abs(y / g.N - x).max() < 1e-12 * np.abs(x).max()


@pytest.mark.gpu
@pytest.mark.parametrize("fp64,nt", [(0, 2048), (0, 4096), (0, 8192), (0, 16384), (0, 32768), (0, 65536),
                                     (1, 2048), (1, 4096), (1, 8192), (1, 16384), (1, 32768)])
def test_bits_do_not_depend_on_the_split(mmp, monkeypatch, fp64, nt):
    prob = W.small_case(seed=400, M=2, nt=nt, n_steps=3, order=8, nnz_target=8)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    outs, ctas = [], []
    for xc in range(max_split(fp64, nt.bit_length() - 1) + 1):
        monkeypatch.setenv("MMP_ROW_SPLIT", str(xc))
        with mmp.Solver(prob) as s:
            s.propagate(3)
            outs.append(s.result())
            ctas.append(s.info()["cluster_ctas"])
    assert ctas == [ctas[0] << i for i in range(len(ctas))]
    assert all(np.array_equal(o, outs[0]) for o in outs)
