"""The transforms' own tables (chl_fft_table) and integer passes, without a GPU:
the passes of the kernels restated over 64-bit integers and run from the
library's table, against numpy.fft; the range that the starting bits promise;
the reciprocals that stand for divisions."""
import numpy as np
import pytest

# even lengths 2^a 3^b up to the longest line that a block's shared memory holds
LENGTHS = sorted({2 ** a * 3 ** b for a in range(1, 13) for b in range(8) if 4 <= 2 ** a * 3 ** b <= 4608})
SIN60 = 0x6ED9EBA16132A9CF


def _words(a):
    """High word and low word >> 1 of 64-bit integers."""
    return a >> 32, (a & 0xFFFFFFFF) >> 1


def _halve(a):
    return (a + ((a >> 1) & 1)) >> 1


def _twiddle(re, im, w, inv):
    """v w / 2 (inverse: v conj(w) / 2) as tw_mul forms it."""
    cx, cy, sx, sy = (w[:, q] for q in range(4))
    r = 0x80000000 + (cx >> 2) + (sx >> 2)
    xh, xl = _words(re)
    yh, yl = _words(im)
    nh, nl = _words(-re if inv else -im)
    ah, al = (yh, yl) if inv else (nh, nl)
    bh, bl = (nh, nl) if inv else (xh, xl)
    t = r + xh * cy + cx * xl + ah * sy + sx * al
    u = r + yh * cy + cx * yl + bh * sy + sx * bl
    return xh * cx + ah * sx + (t >> 31), yh * cx + bh * sx + (u >> 31)


def _sin60(a):
    ah, al = _words(a)
    wh, wl = SIN60 >> 32, (SIN60 & 0xFFFFFFFF) >> 1
    return ((ah * wh) << 1) + ((1409783857 + ah * wl + wh * al) >> 30)


def _butterfly(v, inv):
    s = -1 if inv else 1
    if len(v) == 2:
        (a, b), (c, d) = v
        return [(a + c, b + d), (a - c, b - d)]
    if len(v) == 4:
        ax, ay, bx, by = v[0][0] + v[2][0], v[0][1] + v[2][1], v[0][0] - v[2][0], v[0][1] - v[2][1]
        cx, cy, ex, ey = v[1][0] + v[3][0], v[1][1] + v[3][1], v[1][0] - v[3][0], v[1][1] - v[3][1]
        return [(ax + cx, ay + cy), (bx + s * ey, by - s * ex), (ax - cx, ay - cy), (bx - s * ey, by + s * ex)]
    t0x, t0y = v[1][0] + v[2][0], v[1][1] + v[2][1]
    dx, dy = _sin60(v[1][0] - v[2][0]), _sin60(v[1][1] - v[2][1])
    tx, ty = v[0][0] - _halve(t0x), v[0][1] - _halve(t0y)
    return [(v[0][0] + t0x, v[0][1] + t0y), (tx + s * dy, ty - s * dx), (tx - s * dy, ty + s * dx)]


def _radix(rem):
    return 4 if rem % 4 == 0 else (3 if rem % 3 == 0 else 2)


def passes(N):
    out, rem, Ns = [], N, 1
    while rem > 1:
        R = _radix(rem)
        out.append((R, Ns))
        Ns *= R
        rem //= R
    return out


def transform(re, im, entries, inv):
    """One line through the passes; the largest modulus that a pass with twiddles read."""
    N, top = len(re), 0.0
    P = passes(N)
    tw = len(P)
    for p, (R, Ns) in enumerate(P):
        assert tuple(entries[p, :2]) == (R, Ns)
        nb = N // R
        j = np.arange(nb)
        v = [(re[j + r * nb], im[j + r * nb]) for r in range(R)]
        o, step = j * R, 1
        if p:
            top = max(top, np.hypot(re.astype(float), im.astype(float)).max())
            g, jm = j // Ns, j % Ns
            w = entries.astype(np.int64)
            v[0] = _halve(v[0][0]), _halve(v[0][1])
            for r in range(1, R):
                v[r] = _twiddle(*v[r], w[tw + (r - 1) * Ns + jm], inv)
            tw += Ns * (R - 1)
            o, step = g * Ns * R + jm, Ns
        re, im = np.empty_like(re), np.empty_like(im)
        for r, (a, b) in enumerate(_butterfly(v, inv)):
            re[o + r * step], im[o + r * step] = a, b
    assert tw == len(entries)
    return re, im, top


@pytest.mark.parametrize("N", LENGTHS)
def test_passes_over_the_librarys_table(N):
    """1e-14 of the largest output: a few units of 2^-54 or finer of the line's
    largest component per pass.  Lines that reach the largest modulus at some pass
    (constant in phase with a mode) keep every input of a pass with twiddles below
    2^61, where its sums of four cross products fit."""
    from channel_rl_gb300.host import fft_table
    bits, entries = fft_table(N)
    assert 50 <= bits <= 60
    rng = np.random.default_rng(N)
    big = (1 << bits) - 1
    modes = [0, 1, N // 2, N // 3]
    for inv in (False, True):
        lines = [(rng.integers(-big, big, N), rng.integers(-big, big, N)), (rng.choice((-big, big), N), rng.choice((-big, big), N))]
        for m in modes:
            # the largest square |re|, |im| <= big holds exp(i phase) sqrt(2) big only on its corners
            z = np.exp(2j * np.pi * ((m * np.arange(N)) % N) / N + 0.25j * np.pi)
            lines.append(tuple(np.clip(np.round(a * np.sqrt(2.0)), -1, 1).astype(np.int64) * big for a in (z.real, z.imag)))
        lines.append((np.full(N, big), np.full(N, big)))
        for re, im in lines:
            a, b, top = transform(re.astype(np.int64), im.astype(np.int64), entries, inv)
            assert top < 2.0 ** 61
            x = re.astype(float) + 1j * im.astype(float)
            want = (np.fft.ifft(x) * N if inv else np.fft.fft(x)) * 0.5 ** (len(passes(N)) - 1)
            assert np.abs(a + 1j * b - want).max() <= 1e-14 * max(np.abs(want).max(), float(big))


@pytest.mark.parametrize("N", LENGTHS)
def test_starting_bits_bound_every_pass(N):
    """Modulus: sqrt(2) of the component at the start, times R in the first pass, R/2
    in each later one; none that enters a pass with twiddles reaches 2^61."""
    from channel_rl_gb300.host import fft_table
    m = 2.0 ** fft_table(N)[0] * 2 ** 0.5
    for p, (R, _) in enumerate(passes(N)):
        assert p == 0 or m < 2.0 ** 61
        m *= R if p == 0 else R / 2


def test_reciprocals_divide_exactly():
    from channel_rl_gb300.host import fft_table
    n = np.arange(1 << 16, dtype=np.uint64)
    seen = {}
    for N in LENGTHS:
        for p, (R, Ns) in enumerate(passes(N)):
            for d, m in ((Ns, fft_table(N)[1][p, 2]), (N // R, fft_table(N)[1][p, 3])):
                seen[d] = int(np.uint32(m))
    for d, m in seen.items():
        q = n if m == 0 else (n * np.uint64(m)) >> np.uint64(32)
        assert (q == n // np.uint64(d)).all(), d
        # what the kernels form themselves
        k = 0xFFFFFFFF // d + 1
        assert m == (k if d > 1 else 0)


def test_lengths_without_a_table_are_refused():
    from channel_rl_gb300.host import ChlError, fft_table
    for N in (0, -4, 5, 10, 250):
        with pytest.raises(ChlError):
            fft_table(N)
    assert fft_table(1)[1].shape == (0, 4)
