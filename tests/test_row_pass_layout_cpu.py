"""k_pass_c, the row pass, replayed lane by lane in numpy (CPU only).

The replay follows the kernel's index maps: the even/odd packing and its multipliers, the first
exchange that hands each group of butterflies to adjacent lanes, the padded exchanges inside a
group, the stage multipliers in tensor-memory order, the pixels a lane ends with, the padded
staging of the sums, and, for divided batches, the split into parts and their merge.  It checks

* that a row comes out as the inverse real FFT;
* that every address stays inside its buffer, every element that is read has been written by
  the exchange before (a read of anything else gives NaN), and no element is written twice;
* that 8 lanes of a 16-byte access touch 128 different bytes;
* that the merged maxima and best orientations are those of one pass in order.

The index expressions are looked up in the kernel's source, so that a change there fails here.
"""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cistem_downstream_bah_b200", "csrc",
                   "tm_kernels.cuh")


def _kernel(start, end):
    text = re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", open(SRC).read()))
    return text[text.index(start):text.index(end)]


def test_the_replayed_expressions_are_the_kernels():
    body = _kernel("struct PassC {", "__global__ void k_prepare_image")
    for expr in ("P = H / 8;", "G = P / 8;", "S = P + P / 8;", "ROWS = P >= 128 ? 1 : 128 / P;", "EXL = 8 * S;",
                 "const int jm = (8 * (l + PC::G * u) + j) % Ns;",
                 "p[r] = tw.template w<+1>(jm * (H / (Ns * RS)) * r, H);", "g[2 * (u * (RS - 1) + r - 1)] = p[r].x;",
                 "tmptx::tmem_st16(tcomp + 64, z);", "fill<1>(tcomp + 80, l, j, a.tw)", "fill<2>(tcomp + 96, l, j, a.tw)",
                 "fill<3>(tcomp + 112, l, j, a.tw)", "const int t = tid % P, rl = tid / P;", "const int l = t % G, j = t / G;",
                 "const float2* c = rows + rl * LR + t;", "const float2* d = rows + rl * LR + (P - t);",
                 "hk = c[h * ROWS * LR + P * r], hm = d[h * ROWS * LR + P * (7 - r)];",
                 "put(ex + S * r + t, v[r]);", "float4* const eg = ex + S * j;", "v[r] = get(eg + l + G * r);",
                 "auto pad = [](int e) { return e + (e >> 3); };", "put(eg + 9 * l + r, v[r]);",
                 "v[r] = get(eg + pad(l + G * r));", "const int at = 72 * (l >> 3) + (l & 7);", "put(eg + at + 9 * r, v[r]);",
                 "e[r] = tmfft::pmul(v[u + r * NU], make_float2(tb[2 * i], tb[2 * i + 1]));",
                 "v[u + r * NU] = e[r];", "const int own = rl * X + 16 * l + 2 * j;",
                 "auto pad = [](int e) { return e + (e >> 4); };", "auto px = [pad](int r) { return pad(2 * P * (r / 2)) + r % 2; };",
                 "staged[2 * ROWS * EXL + at + px(r)]", "i0 = part * npairs / parts;", "npairs = (part + 1) * npairs / parts;",
                 "if (p > 0 && mp > m) won = p;", "m = p > 0 ? fmaxf(m, mp) : mp;",
                 "for (int e = part * PER / parts; e < (part + 1) * PER / parts; e++)"):
        assert expr in body, expr


def _plan(H):
    radices = [8, 8]
    while np.prod(radices) < H:
        radices.append(int(min(8, H // np.prod(radices))))
    assert np.prod(radices) == H
    return radices


def _conflict_free(places):
    """places: (lanes,) of 16-byte elements; 8 consecutive lanes touch 8 different ones modulo 8."""
    lanes = places[: len(places) // 8 * 8].reshape(-1, 8) % 8
    return all(len(set(row)) == 8 for row in lanes)


@pytest.mark.parametrize("X", [256, 512, 1024, 2048, 4096])
def test_a_row_is_the_inverse_real_fft(X):
    rng = np.random.default_rng(X)
    H = X // 2
    P, G = H // 8, H // 64
    S = P + P // 8
    radices = _plan(H)
    row = rng.standard_normal(H + 1) + 1j * rng.standard_normal(H + 1)
    t = np.arange(P)
    lane, j = t % G, t // G
    # packing
    v = np.zeros((P, 8), complex)
    for r in range(8):
        hk, hm = row[t + P * r].copy(), row[(P - t) + P * (7 - r)].copy()
        if r == 0:   # the first lane's DC and Nyquist terms, as FFTW's c2r
            hk[0], hm[0] = hk[0].real, hm[0].real
        e, d = hk + hm.conj(), hk - hm.conj()
        v[:, r] = e + 1j * d * np.exp(2j * np.pi * (t + P * r) / X)
    dft8 = np.exp(2j * np.pi * np.outer(np.arange(8), np.arange(8)) / 8)
    v = v @ dft8.T

    def exchange(put, get):
        buf = np.full(8 * S, np.nan, complex)
        count = np.zeros(8 * S, int)
        out = np.empty_like(v)
        for r in range(8):
            place = put(r)
            assert place.min() >= 0 and place.max() < 8 * S
            buf[place] = v[:, r]
            np.add.at(count, place, 1)
            assert _conflict_free(place)
        assert count.max() == 1
        for r in range(8):
            place = get(r)
            assert _conflict_free(place)
            out[:, r] = buf[place]
        assert not np.isnan(out).any()
        return out

    def pad(e):
        return e + (e >> 3)

    v = exchange(lambda r: S * r + t, lambda r: S * j + lane + G * r)
    for s in range(1, len(radices)):
        if s == 2:
            v = exchange(lambda r: S * j + 9 * lane + r, lambda r: S * j + pad(lane + G * r))
        if s == 3:
            v = exchange(lambda r: S * j + 72 * (lane >> 3) + (lane & 7) + 9 * r, lambda r: S * j + pad(lane + G * r))
        RS, Ns = radices[s], int(np.prod(radices[:s]))
        NU = 8 // RS
        cols = np.zeros((P, 16))   # this stage's 16 tensor-memory columns
        for u in range(NU):
            jm = (8 * (lane + G * u) + j) % Ns
            for r in range(1, RS):
                w = np.exp(2j * np.pi * ((jm * (H // (Ns * RS)) * r) % H) / H)
                i = 2 * (u * (RS - 1) + r - 1)
                cols[:, i], cols[:, i + 1] = w.real, w.imag
        dft = np.exp(2j * np.pi * np.outer(np.arange(RS), np.arange(RS)) / RS)
        for u in range(NU):
            e = np.stack([v[:, u + r * NU] for r in range(RS)], 1)
            for r in range(1, RS):
                i = u * (RS - 1) + r - 1
                e[:, r] *= cols[:, 2 * i] + 1j * cols[:, 2 * i + 1]
            e = e @ dft.T
            for r in range(RS):
                v[:, u + r * NU] = e[:, r]
    out = np.full(X, np.nan)
    for r in range(8):
        out[16 * lane + 2 * j + 2 * P * r] = v[:, r].real
        out[16 * lane + 2 * j + 2 * P * r + 1] = v[:, r].imag
    half = row.copy()
    half[0], half[H] = half[0].real, half[H].real
    assert np.allclose(out, np.fft.irfft(half, X) * X, rtol=0, atol=1e-9 * np.abs(out).max())


@pytest.mark.parametrize("X", [256, 512, 1024, 2048, 4096])
def test_sums_are_staged_one_place_per_pixel(X):
    P = X // 16
    rows = 1 if P >= 128 else 128 // P
    G, S = P // 8, P + P // 8
    tid = np.arange(P * rows)
    t, rl = tid % P, tid // P
    own = rl * X + 16 * (t % G) + 2 * (t // G)

    def pad(e):
        return e + (e >> 4)

    places, pixels = [], []
    for r in range(16):
        places.append(pad(own) + pad(2 * P * (r // 2)) + r % 2)
        pixels.append(own + 2 * P * (r // 2) + r % 2)
    places, pixels = np.concatenate(places), np.concatenate(pixels)
    assert sorted(pixels) == list(range(rows * X))
    assert np.array_equal(places, pad(pixels))          # where they are read back, in pixel order
    assert places.max() < 2 * rows * 8 * S               # doubles of half the exchange buffers
    hc = (X // 2 + 1 + 3) // 4 * 4
    boxes = (hc // 4 + 255) // 256
    row_len = 4 * boxes * (((hc // 4 + boxes - 1) // boxes + 3) // 4 * 4)
    assert places.max() < rows * 2 * row_len * 2         # the maxima, floats in the row buffer


@pytest.mark.parametrize("nb,parts", [(8, 2), (9, 2), (16, 4), (17, 4), (33, 8), (41, 8), (128, 8)])
def test_merged_parts_are_one_pass_in_order(nb, parts):
    rng = np.random.default_rng(nb)
    pixels = 512
    values = rng.integers(0, 6, (nb, pixels)).astype(np.float32)    # many equal maxima
    before = rng.integers(-1, 7, pixels).astype(np.float32)
    best0 = np.full(pixels, -7)
    mip, best = before.copy(), best0.copy()
    for o in range(nb):
        better = values[o] > mip
        best[better] = o
        mip = np.maximum(mip, values[o])
    pairs = (nb + 1) >> 1
    covered = []
    maxima, bests = [], []
    for part in range(parts):
        i0, i1 = part * pairs // parts, (part + 1) * pairs // parts
        assert i1 > i0
        m, b = before.copy(), best0.copy() if part == 0 else np.full(pixels, -99)
        for i in range(i0, i1):
            first, second = 2 * i, 2 * i + 1 if 2 * i + 1 < nb else 2 * i   # an odd batch's last twice
            covered += {first, second}
            new = np.maximum(np.maximum(m, values[first]), values[second])
            changed = new > m
            b[changed] = np.where(values[first] == new, first, first + 1)[changed]
            m = new
        maxima.append(m)
        bests.append(b)
    assert sorted(covered) == list(range(nb))
    merged, won = maxima[0].copy(), np.zeros(pixels, int)
    for p in range(1, parts):
        won[maxima[p] > merged] = p
        merged = np.maximum(merged, maxima[p])
    got = np.choose(won, bests)
    assert np.array_equal(merged, mip) and np.array_equal(got, best)
    # a block's share of the 16 pixels per thread
    shares = [e for part in range(parts) for e in range(part * 16 // parts, (part + 1) * 16 // parts)]
    assert shares == list(range(16))
