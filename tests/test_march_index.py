"""Index arithmetic of the marching wavelet kernels (csrc/wavelet.cu: k_wav_analysis_march,
k_wav_synthesis_march and their launchers), replayed on the CPU along each axis: every load
and store lies inside its array and, where a pair is moved, on its boundary; every
tap reads the row or column that the filter bank asks for; every output is made
exactly once, for whole volumes and for column windows, in both output layouts."""
import itertools

import pytest

MW, WARPS = 4, 148 * 32
BANKS = [(10, 4, 2, 4, 2, 10), (2, 0, 2, 0, 2, 2), (8, 0, 8, 0, 8, 8)]  # LL, H0, HN, S0, SN, SH
SIDES = (10, 12, 16, 26, 32, 54, 56, 58, 64, 66, 108, 128, 130)


def segment(length, strips):
    seg = 64
    while seg > 4 and strips * ((length + seg - 1) // seg) < WARPS:
        seg >>= 1
    return seg


def windows(n):
    """(x_lo, x_len) as the launchers take them: all of n columns and circular windows."""
    return [(0, n)] + [(lo, ln) for lo, ln in ((0, 1), (n - 1, min(n, 3)), (n // 2, n - 1)) if ln >= 1]


def analysis_rows(L, shift, W):
    even = shift % 2 == 0
    HL, O = W // 2 if even else W // 2 - 1, L // 2
    nout, made = 32 - HL, []
    for strip in range((O + nout - 1) // nout):
        held = []  # per lane: the logical rows of its pair
        for lane in range(32):
            q = strip * nout - HL + lane
            first = 2 * q if even else 2 * q - 1
            yo = (first - shift) % L
            assert yo % 2 == 0 and yo + 1 < L  # one 8-byte load
            held.append((first, first + 1))
            assert [(r - shift) % L for r in held[-1]] == [yo, yo + 1]
        for lane in range(HL, 32):
            q = strip * nout - HL + lane
            if q >= O:
                continue
            if even:
                v = [held[lane][0]]
                for p in range(1, HL):
                    v += [held[lane - p][1], held[lane - p][0]]
                v += [held[lane - HL][1]]
            else:
                v = [held[lane][1], held[lane][0]]
                for p in range(1, HL + 1):
                    v += [held[lane - p][1], held[lane - p][0]]
            assert v[:W] == [2 * q - k for k in range(W)]
            made.append(q)
    assert sorted(made) == list(range(O))


def analysis_columns(L, shift, W, x_lo, x_len, seg):
    HX, O, U, made = W // 2 - 1, L // 2, W // 2 if W > 2 else 4, []
    assert (2 * U) % W == 0
    for sgi in range((x_len + seg - 1) // seg):
        xs, n = x_lo + sgi * seg, min(seg, x_len - sgi * seg)
        xc, ox = (2 * (xs - HX) - 1 - shift) % L, xs - O if xs >= O else xs
        ring = {}
        for t in range(n + HX):
            u = t % U
            for c in range(2):
                assert 0 <= xc < L
                ring[(2 * u + c) % W] = xc
                xc = 0 if xc + 1 == L else xc + 1
            if t >= HX:
                assert 0 <= ox < O
                for k in range(W):
                    assert ring[(2 * u + 1 - k) % W] == (2 * ox - k - shift) % L
                made.append(ox)
                ox = 0 if ox + 1 == O else ox + 1
    assert sorted(made) == sorted((x_lo + x) % O for x in range(x_len))


def synthesis_taps(S0, SN, SH):
    """(output parity, tap, offset of the coefficient it reads), as both passes write them."""
    for k in itertools.chain(range(S0, S0 + SN), range(SH)):
        yield (0, k, k // 2) if k % 2 == 0 else (1, k, (k + 1) // 2)


def synthesis_rows(L, shift, S0, SN, SH, gs):
    W = max(S0 + SN, SH)
    HS, I, PQ, made = W // 2, L // 2, 40, []
    assert 32 + HS <= PQ and 8 * HS <= 64
    for strip in range((I + 31) // 32):
        q0, ring = strip * 32, {}
        for lane in range(32):
            ring[lane] = (q0 + lane) % I  # of every band
            for h in range(2):
                e = lane + 32 * h
                if e < 8 * HS:
                    assert 0 <= e // HS < 8
                    ring[32 + e % HS] = (q0 + 32 + e % HS) % I
        assert set(ring) == set(range(32 + HS))
        for lane in range(32):
            q = q0 + lane
            if q >= I:
                continue
            for par, k, off in synthesis_taps(S0, SN, SH):
                assert off <= HS and ring[lane + off] == ((2 * q + par + k) // 2) % I
                assert (2 * q + par + k) % 2 == 0
            rows = [(2 * q + p - shift) % L for p in range(2)]
            at = [((r >> gs) << (2 * gs)) + (r & ((1 << gs) - 1)) if gs else r for r in rows]  # one slot
            if shift % 2 == 0:
                assert at[0] % 2 == 0 and at[1] == at[0] + 1  # one 8-byte store
            made += rows
    assert sorted(made) == list(range(L))


def synthesis_columns(L, Oy, Oz, shift, S0, SN, SH, x_lo, x_len, seg, gs):
    HS, I, NST, made = max(S0 + SN, SH) // 2, L // 2, 4, []
    step = Oy if gs == 0 else ((Oy >> gs) * Oz) << (2 * gs)
    mask = (1 << gs) - 1

    def address(x):
        return (x >> gs) * step + ((x & mask) << gs)

    def after(x, c):
        return 0 if x + 1 == L else c + (1 << gs) if (x + 1) & mask else ((x + 1) >> gs) * step

    for sgi in range((x_len + seg - 1) // seg):
        xs, n = x_lo + sgi * seg, min(seg, x_len - sgi * seg)
        T, xc, staged, window = n + HS, xs - I if xs >= I else xs, {}, []
        ox = (2 * xs - shift) % L
        col = address(ox)

        def stage(slot):
            nonlocal xc
            assert 0 <= xc < I
            staged[slot] = xc
            xc = 0 if xc + 1 == I else xc + 1

        for p in range(NST - 1):
            if p < T:
                stage(p)
        for t in range(T):
            if t + NST - 1 < T:
                stage((t + NST - 1) % NST)
            window = (window + [staged[t % NST]])[-(HS + 1):]
            cols = [col, after(ox, col)]
            if t >= HS:
                j = xs + t - HS
                for par, k, off in synthesis_taps(S0, SN, SH):
                    assert window[off] == ((2 * j + par + k) // 2) % I
                for par in range(2):
                    x = (2 * j + par - shift) % L
                    assert cols[par] == address(x)
                    made.append(x)
                ox = 0 if ox + 1 == L else ox + 1
                col = after(ox, cols[1])
                ox = 0 if ox + 1 == L else ox + 1
    assert sorted(made) == sorted((2 * (x_lo + x) + p - shift) % L for x in range(x_len) for p in range(2))


@pytest.mark.parametrize("bank", BANKS)
def test_march_analysis(bank):
    LL, H0, HN = bank[:3]
    W = max(LL, H0 + HN)
    for L in SIDES + ((2, 4, 6, 8) if W == 2 else (8,) if W == 8 else ()):
        for shift in (0, 1, 2, 3, 7, L + 1):
            analysis_rows(L, shift, W)
            for lo, ln in windows(L // 2):
                for strips in (1, 60, 5000):
                    analysis_columns(L, shift, W, lo, ln, segment(ln, strips))


@pytest.mark.parametrize("bank", BANKS)
def test_march_synthesis(bank):
    S0, SN, SH = bank[3:]
    W = max(S0 + SN, SH)
    for L in SIDES + ((2, 4, 6, 8) if W == 2 else (8,) if W == 8 else ()):
        for shift, gs in itertools.product((0, 1, 2, 3, 7, L + 1), (0, 3, 4)):
            if gs and L % (1 << gs):
                continue
            synthesis_rows(L, shift, S0, SN, SH, gs)
            for lo, ln in windows(L // 2):
                for strips in (1, 5000):
                    synthesis_columns(L, 32, 8, shift, S0, SN, SH, lo, ln, segment(ln, strips), gs)
