"""Index algebra of the level-paired line transforms (csrc/zfft.cuh, zfft.cu),
restated here: the factorisation of a line, its padded in-place positions, the
digit-reversed rows of the adjacent pass, the butterfly pairs of the pass that
works on wavenumbers k and N - k, and the split of a packed level pair.  Every
position stays inside the line's buffer, every one is written once per pass, and
the passes give the discrete Fourier transform, for every even length whose half
has no factor above 5 (the lengths a plan takes).
"""
import numpy as np
import pytest

EDGE = (8, 4, 9, 10, 6, 5, 3, 2)
MID = (16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2)
LAST = (8, 6, 4, 2)


def factors(N, elem):
    """zplan_make: the cheapest factorisation (adjacent, middle.., last)."""
    best = None

    def consider(r):
        nonlocal best
        c = 100.0 * len(r)
        for i, q in enumerate(r):
            last = i == len(r) - 1
            c += abs(q - (4 if last and elem == 8 else 8)) * (2.0 if i == 0 or last else 1.0)
        if r[0] not in (8, 4) and r[0] % 2 == 0:
            c += 8
        if r[0] == 10:
            c += 4
        if best is None or c < best[0]:
            best = (c, r)

    for a in EDGE:
        for z in LAST:
            if N % (a * z):
                continue
            m = N // (a * z)
            if m == 1:
                consider((a, z))
                continue
            for b in MID:
                if m % b:
                    continue
                if m == b:
                    consider((a, b, z))
                else:
                    for c in MID:
                        if m == b * c:
                            consider((a, b, c, z))
    return best and best[1]


class Line:
    def __init__(self, N, elem):
        self.N, self.r = N, factors(N, elem)
        self.S = [int(np.prod(self.r[:i])) for i in range(len(self.r))]
        self.Q = N // self.r[-1]
        self.sh = {2: 1, 4: 2, 8: 3}.get(self.r[0], 31)
        self.NP = N + (N >> self.sh)

    def phys(self, pos):
        return pos + (pos >> self.sh)

    def rev(self, b):
        acc = 0
        for R in self.r[1:]:
            acc, b = acc * R + b % R, b // R
        return acc


def lengths(lo, hi):
    out = []
    for n in range(lo, hi + 1, 2):
        m = n // 2
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def forward(L, x):
    """Decimation in time, in place: rows in, natural wavenumbers out."""
    N, buf = L.N, np.full(L.NP, np.nan, complex)
    R = L.r[0]
    for b in range(N // R):
        pos = L.phys(b * R) + np.arange(R)  # adjacent slots
        assert all(np.isnan(buf[pos].real)) and pos.max() < L.NP
        buf[pos] = np.fft.fft(x[L.rev(b) + (N // R) * np.arange(R)])
    for i in range(1, len(L.r)):
        R, S, seen = L.r[i], L.S[i], set()
        for b in range(N // R):
            m, k = divmod(b, S)
            base = L.phys(m * S * R + k)
            pos = base + np.arange(R) * (S + (S >> L.sh))
            assert list(pos) == [L.phys(m * S * R + k + j * S) for j in range(R)]
            assert pos.max() < L.NP and not seen & set(pos)
            seen |= set(pos)
            w = np.exp(-2j * np.pi * np.arange(R) * k * (N // (S * R)) / N)
            buf[pos] = np.fft.fft(buf[pos] * w)
    return np.array([buf[L.phys(k)] for k in range(N)])


def inverse(L, F):
    """Decimation in frequency, in place: natural wavenumbers in, rows out."""
    N, buf = L.N, np.full(L.NP, np.nan, complex)
    for k in range(N):
        buf[L.phys(k)] = F[k]
    for i in range(len(L.r) - 1, 0, -1):
        R, S = L.r[i], L.S[i]
        for b in range(N // R):
            m, k = divmod(b, S)
            pos = L.phys(m * S * R + k) + np.arange(R) * (S + (S >> L.sh))
            w = np.exp(2j * np.pi * np.arange(R) * k * (N // (S * R)) / N)
            buf[pos] = np.fft.ifft(buf[pos]) * R * w
    out, R = np.empty(N, complex), L.r[0]
    for b in range(N // R):
        pos = L.phys(b * R) + np.arange(R)
        out[L.rev(b) + (N // R) * np.arange(R)] = np.fft.ifft(buf[pos]) * R
    return out


def pairs(L):
    """Butterfly pairs (t1, t2) of the last pass, t2 None where t1 has no partner."""
    for s in range((L.Q + 1) // 2):
        yield (s, L.Q - s) if s else (0, None if L.Q % 2 else L.Q // 2)


@pytest.mark.parametrize("elem", [4, 8])
def test_every_length_has_a_line_and_its_passes_are_the_transform(elem):
    rng = np.random.default_rng(5)
    done = 0
    for N in lengths(4, 1100):
        if factors(N, elem) is None:
            assert N < 8  # shorter lines keep the other kernels
            continue
        L = Line(N, elem)
        assert int(np.prod(L.r)) == N and L.r[-1] % 2 == 0 and len(L.r) <= 4
        if N > 300 and N % 64 and N % 45:
            continue  # the algebra of every fourth or so of the long ones
        x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
        ref = np.fft.fft(x)
        # 1e-13 is 450 ulp of the rms, over the log2(N) <= 10 rounding stages
        assert np.abs(forward(L, x) - ref).max() <= 1e-13 * np.sqrt(N) * np.abs(x).max()
        assert np.abs(inverse(L, ref) / N - x).max() <= 1e-13 * np.sqrt(N) * np.abs(x).max()
        done += 1
    assert done > 40


@pytest.mark.parametrize("N", [8, 50, 96, 162, 250, 384, 1024])
def test_the_pairs_of_the_last_pass_give_both_levels_half_spectra(N):
    L, R = Line(N, 4), Line(N, 4).r[-1]
    a, b = np.random.default_rng(N).standard_normal((2, N))
    F = np.fft.fft(a + 1j * b)
    A, B, seen = np.fft.fft(a), np.fft.fft(b), []
    for t1, t2 in pairs(L):
        idx = [(t1 + L.Q * j, None) for j in range(R // 2 + (t1 == 0))]
        if t2 is not None:
            idx += [(t2 + L.Q * j, None) for j in range(R // 2)]
        for k, _ in idx:
            f, g = F[k], F[(N - k) % N]
            # the partner comes from the pair's own butterflies
            assert (N - k) % N % L.Q in (t1, t2)
            xa = 0.5 * complex(f.real + g.real, f.imag - g.imag)
            xb = 0.5 * complex(f.imag + g.imag, g.real - f.real)
            assert abs(xa - A[k]) <= 1e-12 * N and abs(xb - B[k]) <= 1e-12 * N
            # and back: both packed wavenumbers from the two half spectra
            assert abs(complex(xa.real - xb.imag, xa.imag + xb.real) - f) <= 1e-12 * N
            assert abs(complex(xa.real + xb.imag, xb.real - xa.imag) - g) <= 1e-12 * N
            seen.append(k)
    assert sorted(seen) == list(range(N // 2 + 1))
