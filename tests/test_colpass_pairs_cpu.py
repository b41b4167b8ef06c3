"""k_pass_b_rg, the residue-grouped column pass on column pairs (height 4096, 256-row templates),
replayed thread by thread in numpy, and the shared-memory places of k_pass_b's transforms (CPU only).

The replay of one item (four columns of one orientation, 512 threads, two adjacent columns each)
follows the kernel's index maps: staging of the rows of A, the residue twiddles and I' in the order
of the transforms' groups of four, the transposes through the warp's own buffers, the block
buffer, and the output tiles that are built in place.  It checks the item against the FFT
definition, C's tiles against the kernels' own layout function, every address against its buffer, and
that 8 lanes of an access touch different banks.  The index expressions are looked up in the
kernel's source, so that a change there fails here.

For k_pass_b the C++ plan itself is compiled for the host: every transform's places lie inside the
buffer, no two elements share one, and the split of a place into a base and a compile-time offset is exact
wherever the kernel uses it.
"""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cistem_downstream_bah_b200", "csrc")
Y, T, NT, RS = 4096, 256, 512, 17
SCR = 16 * RS + 8


def _kernel(start, end):
    text = open(os.path.join(CSRC, "tm_kernels.cuh")).read()
    text = re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", text))
    return text[text.index(start):text.index(end)]


def test_the_replayed_expressions_are_the_kernels():
    body = _kernel("struct PassBRg {", "inline int hist_copies")
    for expr in ("static constexpr int RS = 17;", "static constexpr int SCR = 16 * RS + 8;", "W = 4, NT = 512;",
                 "sizeof(float4) * 16 * 256 * 2;", "sizeof(float2) * 16 * 2 * SCR;", "sizeof(float4) * 2 * T;",
                 "(size_t)(tid >> 1) * a.XP + 2 * (tid & 1);", "tmptx::smem_u32(abuf + tid);",
                 "const int s = tid >> 5, q = (tid >> 1) & 15, cp = tid & 1;",
                 "const int r = 2 * h + i / 4 + 4 * (i % 4);", "a.twy.template w<-1>((q + 16 * r) * s, Y);",
                 "a.twy.template w<-1>(16 * q, Y)", "a.Ip + (size_t)(s + 16 * q) * a.XP + group * 4 + 2 * cp",
                 "__ldg(Ig + (size_t)(128 * (h + 4 * r)) * a.XP);", "+ (2 * s + cp) * PB::SCR;",
                 "const float4* ac = abuf + (it & 1) * (2 * T) + (tid & 31);", "ac[32 * (g + 4 * k)];",
                 "scr[RS * q + g + 4 * k] = v[4 * g + k].re;", "scr[RS * q + g + 4 * k] = v[g + 4 * k].re;",
                 "im[r] = v[4 * (r % 4) + r / 4].im;", "v[r].re = scr[RS * r + q];", "v[g + 4 * k].im = scr[RS * (g + 4 * k) + q];",
                 "put(blk + (s * 256 + q + 16 * (i / 4 + 4 * (i % 4))) * 2 + cp, v[i]);", "get(blk + 512 * (g + 4 * k) + tid);",
                 "blk[512 * (g + 4 * k) + tid] = make_float4(z.re.x, z.im.x, z.re.y, z.im.y);",
                 "tmptx::tensor3_s2g(&cmap, 0, group, o * (Y / 8), blk);",
                 "tmptx::tensor3_s2g(&cmap, 0, group, o * (Y / 8) + 256, blk + 4096);"):
        assert expr in body, expr


def _dft4(v, i, sign):
    v[..., i] = v[..., i] @ np.exp(sign * 2j * np.pi * np.outer(np.arange(4), np.arange(4)) / 4)


def _mid(v, sign):
    for a in range(4):
        for b in range(4):
            v[..., 4 * a + b] *= np.exp(sign * 2j * np.pi * a * b / 16)


def _level1(v, g, sign):
    _dft4(v, [g, 4 + g, 8 + g, 12 + g], sign)


def _level2(v, g, sign):
    _dft4(v, [4 * g, 4 * g + 1, 4 * g + 2, 4 * g + 3], sign)


class _Shared:
    """A buffer of pairs of columns: written once per element, read only where written."""

    def __init__(self, size, banks):
        self.data, self.banks = np.full((size, 2), np.nan, complex), banks

    def _check(self, at):
        assert at.min() >= 0 and at.max() < len(self.data)
        lanes = at.reshape(-1, self.banks) % self.banks
        assert all(len(set(row)) == self.banks for row in lanes)

    def write(self, places, values):   # (lanes, 16), (2, lanes, 16)
        assert len(np.unique(places)) == places.size
        for r in range(16):
            self._check(places[:, r])
        self.data[places] = np.moveaxis(values, 0, -1)

    def read(self, places):
        for r in range(16):
            self._check(places[:, r])
        out = np.moveaxis(self.data[places], -1, 0)
        assert not np.isnan(out).any()
        return out


def _replay(A, Ip):
    """A: (256, 4), Ip: (4096, 4) -> the block buffer as float4 elements, (8192, 2) complex."""
    tid = np.arange(NT)
    s, q, cp = tid >> 5, (tid >> 1) & 15, tid & 1
    r16 = np.arange(16)
    abuf = _Shared(2 * T, 8)
    abuf.data[tid] = A[(tid >> 1)[:, None], 2 * (tid & 1)[:, None] + np.arange(2)]

    def table(h_of):   # 16 columns in groups of four, two groups per half
        order = np.empty(16, int)
        for h in range(2):
            for i in range(8):
                order[8 * h + i] = 2 * h + i // 4 + 4 * (i % 4)
        return order

    order = table(None)   # place 4 g + k holds r = g + 4 k
    assert np.array_equal(order, [g + 4 * k for g in range(4) for k in range(4)])
    wres = np.exp(-2j * np.pi * ((q[:, None] + 16 * order) * s[:, None]) / Y)
    wq = np.exp(-2j * np.pi * (q[:, None] * order) / 256)
    iprime = np.empty((2, NT, 16), complex)   # place 4 h + r: I' of k = s + 16 q + 256 (h + 4 r)
    for h in range(4):
        for r in range(4):
            # float4 steps of 128 (h + 4 r) XP are 256 (h + 4 r) rows
            row = s + 16 * q + 256 * (h + 4 * r)
            for c in range(2):
                iprime[c, :, 4 * h + r] = Ip[row, 2 * cp + c]
    v = np.empty((2, NT, 16), complex)
    lane = tid & 31
    for g in range(4):
        for k in range(4):
            v[..., g + 4 * k] = abuf.data[lane + 32 * (g + 4 * k)].T * wres[:, 4 * g + k]
    for g in range(4):
        _level1(v, g, -1)
    _mid(v, -1)
    for g in range(4):
        _level2(v, g, -1)
        v[..., 4 * g:4 * g + 4] *= wq[:, 4 * g:4 * g + 4]
    scr_base = (2 * s + cp) * SCR
    gk = np.array([g + 4 * k for g in range(4) for k in range(4)])   # column of value 4 g + k

    def transpose(v, columns):
        # (real and imaginary parts go one after the other through the same places: 8 bytes each)
        scr = _Shared(16 * 2 * SCR, 16)
        scr.write(scr_base[:, None] + RS * q[:, None] + columns, v)
        return scr.read(scr_base[:, None] + RS * r16 + q[:, None])

    v = transpose(v, gk)
    for g in range(4):
        _level1(v, g, -1)
    _mid(v, -1)
    for g in range(4):
        _level2(v, g, -1)                      # value 4 g + k: k2 = g + 4 k
        v[..., 4 * g:4 * g + 4] = iprime[..., 4 * g:4 * g + 4] * v[..., 4 * g:4 * g + 4].conj()
        _level2(v, g, +1)                      # the inverse's first level takes the same four
    # the factors are symmetric: values stay where level 1 left them
    _mid(v, +1)
    for g in range(4):
        _level1(v, g, +1)
        for k in range(4):
            v[..., g + 4 * k] *= wq[:, 4 * g + k].conj()
    v = transpose(v, r16)                      # value g + 4 k: column m1 = g + 4 k
    for g in range(4):
        _level1(v, g, +1)
    _mid(v, +1)
    for g in range(4):
        _level2(v, g, +1)
        v[..., 4 * g:4 * g + 4] *= wres[:, 4 * g:4 * g + 4].conj()
    blk = _Shared(16 * 256 * 2, 8)
    places = np.stack([(s * 256 + q + 16 * (i // 4 + 4 * (i % 4))) * 2 + cp for i in range(16)], 1)
    blk.write(places, v)
    v = blk.read(tid[:, None] + 512 * r16)
    for g in range(4):
        _level1(v, g, +1)
    _mid(v, +1)
    for g in range(4):
        _level2(v, g, +1)
    out = _Shared(16 * 256 * 2, 8)
    out.write(tid[:, None] + 512 * gk, v)
    return out.data


def test_an_item_is_the_column_pass():
    rng = np.random.default_rng(5)
    A = rng.standard_normal((T, 4)) + 1j * rng.standard_normal((T, 4))
    Ip = rng.standard_normal((Y, 4)) + 1j * rng.standard_normal((Y, 4))
    blk = _replay(A, Ip)
    F = np.fft.fft(A, Y, axis=0)
    want = np.fft.ifft(Ip * F.conj(), axis=0) * Y
    # the buffer is the item's tiles: 8 rows x 4 columns, two float4 (column pairs) a row
    y, kx = np.meshgrid(np.arange(Y), np.arange(4), indexing="ij")
    place = (y // 8) * 32 + (y % 8) * 4 + kx   # c_index of one column group
    got = blk.reshape(-1)[place]
    assert np.allclose(got, want, rtol=0, atol=1e-9 * np.abs(want).max())


PROGRAM = r"""
#include "tm_kernels.cuh"
#include <cstdio>
#include <utility>
#include <vector>

// stage s writes every element once, at the base plus the compile-time offset under pfft's condition
template <int L, int R, int D, int s>
static int stage() {
    using PL = tmfft::Plan<L, R>;
    constexpr int RS = PL::radix(s), Ns = PL::ns(s);
    std::vector<int> hit(L, 0);
    for (int b = 0; b < L / RS; b++) {
        const int idxD = (b / Ns) * Ns * RS + b % Ns;
        for (int r = 0; r < RS; r++) {
            if (idxD + r * Ns >= L || hit[idxD + r * Ns]++) return 3;
            if ((D == 0 || Ns % (D ? D : 1) == 0 || (Ns == 1 && D % RS == 0)) &&
                tmfft::pad_at<D>(idxD) + tmfft::pad_at<D>(r * Ns) != tmfft::pad_at<D>(idxD + r * Ns)) return 4;
        }
    }
    return 0;
}
template <int L, int R, int D, int... s>
static int stages(std::integer_sequence<int, s...>) {
    int e = 0;
    (void)((e = stage<L, R, D, s>()) || ...);
    return e;
}
// the places of one transform of length L in a buffer of `size` elements: inside it, one per element, and
// equal to the base plus the compile-time offset under the conditions of tmfft::pfft
template <int L, int R, int D>
static int transform(int size) {
    using PL = tmfft::Plan<L, R>;
    constexpr int P = PL::P, N = PL::stages;
    std::vector<int> seen(size, 0);
    for (int i = 0; i < L; i++) {
        const int at = tmfft::pad_at<D>(i);
        if (at < 0 || at >= size || seen[at]++) return 1;
    }
    if (D == 0 || P % (D ? D : 1) == 0 || D % P == 0)
        for (int t = 0; t < P; t++)
            for (int r = 0; r < R; r++) {
                const int base = D % P == 0 && P < D ? t : tmfft::pad_at<D>(t);
                if (base + tmfft::pad_at<D>(P * r) != tmfft::pad_at<D>(t + P * r)) return 2;
            }
    return stages<L, R, D>(std::make_integer_sequence<int, N - 1>());
}

template <int T, int Y>
static int pass() {
    using PB = tmk::PassB<T, Y>;
    if (const int e = transform<Y, PB::V, PB::D>(PB::CS)) return e;
    if (const int e = transform<PB::L, PB::V, PB::DF>(PB::RST)) return 10 + e;   // each region
    if (PB::MY * PB::RST > PB::CS) return 21;
    if (PB::EXCH != sizeof(float4) * PB::WP * PB::CS || PB::SMEM > 232448) return 22;
    // the threads' butterflies: every residue's, once
    std::vector<int> seen(PB::P, 0);
    for (int j = 0; j < PB::P; j++) {
        const int s = j % PB::MY, tp = j / PB::MY;
        if (tp >= PB::PT || seen[s * PB::PT + tp]++) return 23;
    }
    // the output's addresses: rows j + P r of a column from those of r = 0 and 1
    const int XP = 12;
    for (int j = 0; j < PB::P; j++)
        for (int r = 0; r < PB::V; r++) {
            const size_t c0 = tmk::c_index<Y>(3, j, 4, XP);
            const size_t c1 = PB::P % tmk::c_tile_rows(Y) == 0 ? c0 + (size_t)PB::P * XP : tmk::c_index<Y>(3, j + PB::P, 4, XP);
            if ((r % 2 ? c1 : c0) + (size_t)(r / 2) * 2 * PB::P * XP != tmk::c_index<Y>(3, j + PB::P * r, 4, XP)) return 24;
        }
    return 0;
}

#define CHECK(T, Y) if (const int e = pass<T, Y>()) return std::printf("FAIL template %d, height %d: %d\n", T, Y, e), 1;
int main() {
    CHECK(32, 256) CHECK(32, 512) CHECK(64, 512) CHECK(64, 1024) CHECK(128, 1024) CHECK(128, 2048) CHECK(256, 2048)
    CHECK(256, 4096) CHECK(64, 4096) CHECK(32, 288) CHECK(48, 256) CHECK(48, 288) CHECK(256, 3888) CHECK(256, 5832)
    CHECK(384, 4096) CHECK(384, 5832) CHECK(128, 4096) CHECK(128, 3888) CHECK(128, 5832) CHECK(64, 3888) CHECK(64, 5832)
    CHECK(384, 3888) CHECK(256, 2916) CHECK(128, 2916) CHECK(256, 1944) CHECK(256, 2592) CHECK(256, 5184) CHECK(64, 256)
    CHECK(128, 256) CHECK(256, 512)
    std::printf("OK\n");
    return 0;
}
"""


def test_places_of_the_stockham_pass(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "places.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "places"
    # the header's device code is compiled for sm_100a as in the library; only host code runs
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--extended-lambda", "-I", CSRC,
                    "-o", str(exe), str(src)], check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout
