"""Index arithmetic of the streaming FFT pass (fft_stream_kernel, csrc/fft.cu)
on the CPU, for every shape it is instantiated with: shared-memory indices
inside their regions, 16-byte accesses aligned, every word of a column loaded
and stored exactly once per pass, every exchange a permutation, and every
twiddle equal to the layer's group twiddle."""
import numpy as np
import pytest

CONTIGUOUS = [(L, 0, 12) for L in range(5, 13)] + [(13, 0, 13)]
STRIDED = [(5, 7, 12), (6, 6, 12), (7, 5, 12), (8, 4, 12), (9, 4, 13)]
R, NQ = 5, 32


def in_pad(e, inv, C):
    return e + 4 * (e >> 5) + 8 * (e >> 8) if inv and C == 0 else e + 4 * (e >> 7)


def padw(e):
    return e + (e >> 5)


def stages(inv, L, C, T):
    K = (L + R - 1) // R
    out = []
    for k in range(K):
        if inv:
            s0 = C + k * R if k + 1 < K else T - R
            ja, jb = (0 if k + 1 < K else C + k * R - s0), R
        else:
            s0 = T - (k + 1) * R if k + 1 < K else C
            ja, jb = 0, (R if k + 1 < K else T - k * R - C)
        out.append((s0, ja, jb))
    return out


@pytest.mark.parametrize("inv", [False, True])
@pytest.mark.parametrize("L,C,TB", CONTIGUOUS + STRIDED)
def test_stream_pass_indices(inv, L, C, TB):
    T = TB if C else L
    threads = 1 << (TB - 5)
    tid = np.arange(threads)
    q = np.arange(NQ)
    words = 1 << TB
    in_words = in_pad(words, inv, C)
    two = not inv and C == 0  # a second buffer for the exchanges
    x_words = words // 8 * 9 if two else in_words
    tw_words = 1 << L if C else 1 << (TB - 1)
    # arriving tile: 16-byte chunks, aligned, inside the region, each word once
    e = (4 * tid[:, None] + 4 * threads * np.arange(8)).ravel()
    d = in_pad(e, inv, C)
    assert np.array_equal(d, (in_pad(4 * tid, inv, C)[:, None] + in_pad(4 * threads * np.arange(8), inv, C)).ravel())
    assert np.all(d % 4 == 0) and d.max() + 4 <= in_words
    assert np.unique((d[:, None] + np.arange(4)).ravel()).size == words
    assert np.array_equal(np.sort((e[:, None] + np.arange(4)).ravel()), np.arange(words))
    layers = []
    for k, (s0, ja, jb) in enumerate(stages(inv, L, C, T)):
        ebase = ((tid >> s0) << (s0 + R)) | (tid & ((1 << s0) - 1))
        el = ebase[:, None] | (q << s0)
        assert np.array_equal(np.sort(el.ravel()), np.arange(words))
        assert s0 >= C
        if k == 0:
            assert np.array_equal(in_pad(ebase, inv, C)[:, None] + in_pad(q << s0, inv, C), in_pad(el, inv, C))
            if inv and C == 0:  # 8 16-byte loads of 32 consecutive words
                assert s0 == 0 and np.array_equal(in_pad(el, inv, C), in_pad(ebase, inv, C)[:, None] + q)
        pad = padw if two else lambda v: in_pad(v, inv, C)
        px = pad(ebase)[:, None] + pad(q << s0)
        assert np.array_equal(px, pad(el)) and px.max() < x_words and np.unique(px).size == words
        grp = tid >> s0
        for j in range(ja, jb):
            layer = s0 + j - C
            layers.append(layer)
            cnt = 1 << (R - 1 - j)
            rows = (el >> C)[:, [v for v in range(NQ) if not v & (1 << j)]]
            group = rows >> (layer + 1)  # within the tile (the chunk, in a contiguous pass)
            mine = (grp << (R - 1 - j))[:, None] + np.array([v >> (j + 1) for v in range(NQ) if not v & (1 << j)])
            assert np.array_equal(group, mine)
            if C == 0 and layer == 0:
                sec = 1 << (TB - 2)  # layer 1's section: 8 twiddles per thread
                assert s0 == 0 and (sec + 8 * grp).max() + 8 <= 2 * sec <= tw_words and np.all((sec + 8 * grp) % 4 == 0)
                continue
            sec = 1 << ((L if C else TB) - 1 - layer)
            first = sec + (grp << (R - 1 - j))
            assert first.max() + cnt <= 2 * sec <= tw_words
            assert np.all(first % min(cnt, 4) == 0)
    assert sorted(layers) == list(range(L))
    if not inv and C == 0:  # stores through shared memory, rows of 32 words and 4 of padding
        assert stages(inv, L, C, T)[-1][0] == 0 and 36 * (threads - 1) + 32 <= x_words
        e = 4 * tid[:, None] + 4 * threads * np.arange(8)
        assert np.array_equal(e + 4 * (e >> 5), 36 * (e >> 5) + (e & 31))


def circle_rule(n, i, h, tw_len):
    """Index of layer i's twiddle for group h (i >= 1) in the tree."""
    return tw_len - (1 << (n - i)) + h


@pytest.mark.parametrize("n,lo,L,C,TB", [(12, 0, 12, 0, 12), (13, 0, 13, 0, 13), (18, 0, 9, 0, 12), (18, 9, 9, 4, 13),
                                        (20, 9, 9, 4, 13), (19, 11, 8, 4, 12), (17, 12, 5, 7, 12), (20, 0, 6, 0, 12),
                                        (16, 10, 6, 6, 12), (21, 14, 7, 5, 12), (26, 0, 10, 0, 12)])
def test_stream_pass_twiddle_sections(n, lo, L, C, TB):
    """The block's table holds, at section + local group, the layer's twiddle of
    that group, for the first, a middle and the last set; columns are covered."""
    tw_len = 1 << (n - 1)
    n_sets = 1 << (n - lo - L if C else n - TB)
    for st in {0, n_sets // 2, n_sets - 1}:
        for lg in range(L if C else TB - 1):
            if not C and lg < TB - L:
                continue
            loc = np.array([0, (1 << lg) - 1])
            src = tw_len - (1 << (n - lo - (L - 1) + lg if C else n - (TB - 1) + lg)) + (st << lg) + loc
            layer = lo + L - 1 - lg if C else TB - 1 - lg
            # group of a word whose rows (words) in the tile give the local group
            v = (st << (lo + L)) + (loc << (layer + 1)) if C else (st << TB) + (loc << (layer + 1))
            assert np.array_equal(src, circle_rule(n, layer, v >> (layer + 1), tw_len))
            assert src.max() < tw_len and src.min() >= 0 and layer >= 1
    if C:  # sets x middle indices x rows x row words tile the column
        mids = 1 << (lo - C)
        assert n_sets * mids << (L + C) == 1 << n
        row = np.arange(1 << L)
        some = [(s << (lo + L)) | (m << C) | (row << lo) for s in {0, n_sets - 1} for m in {0, mids - 1}]
        assert max(x.max() for x in some) + (1 << C) <= 1 << n
        assert all(np.all(x % 4 == 0) for x in some)


@pytest.mark.parametrize("L,C,TB", STRIDED)
@pytest.mark.parametrize("ext", [0, 1, 3])
def test_stream_pass_addresses_step(L, C, TB, ext):
    """Row steps from one address, the mask on the tile's base alone, give the
    masked word of every 16-byte load; byte offsets of the stores fit 32 bits."""
    threads = 1 << (TB - 5)
    tid = np.arange(threads)
    for lo in {C, C + 1, 13, 30 - ext - L}:
        coeff, n = lo + L, lo + L + ext
        mask = (1 << coeff) - 1
        sets, mids = 1 << ext, 1 << (lo - C)
        for st in {0, sets - 1}:
            for mid in {0, mids - 1}:
                base = (st << (lo + L)) | (mid << C)
                e0 = 4 * tid
                p = (base & mask) | ((e0 >> C) << lo) | (e0 & ((1 << C) - 1))
                for k in range(8):
                    e = e0 + 4 * threads * k
                    v = base | ((e >> C) << lo) | (e & ((1 << C) - 1))
                    assert np.array_equal(v & mask, p + k * ((4 * threads >> C) << lo))
                for s0, _, _ in (stages(False, L, C, TB)[-1], stages(True, L, C, TB)[-1]):
                    ebase = ((tid >> s0) << (s0 + R)) | (tid & ((1 << s0) - 1))
                    at = 4 * (base | ((ebase >> C) << lo) | (ebase & ((1 << C) - 1)))
                    for k in range(NQ):
                        e = ebase | (k << s0)
                        v = base | ((e >> C) << lo) | (e & ((1 << C) - 1))
                        assert np.array_equal(at + k * (4 << (s0 - C + lo)), 4 * v) and v.max() < 1 << n
                        assert 4 * v.max() < 1 << 32


def test_butterflies_on_centred_twiddles():
    """bfly_fwd / bfly_inv in 32-bit words at the edges of their ranges and at
    random: both forms of the operands, results within their ranges and equal
    to the butterfly mod p."""
    P, M = 2**31 - 1, 2**32
    edge = np.array([0, 1, 2, P - 1, P - 2, 2**30, 2**30 - 1, 2**30 + 1, 2**16], dtype=object)
    rng = np.random.default_rng(3)
    rand = np.array([int(v) for v in rng.integers(0, P, 9)], dtype=object)
    vals = np.concatenate([edge, rand])
    a, b, w = (g.ravel() for g in np.meshgrid(vals, vals, vals, indexing="ij"))
    signed = lambda x: np.where(x >= M // 2, x - M, x)

    def mul_centred(x, s):
        p = signed(x) * signed(s) + 2**31 - 2**62
        assert p.min() >= -2**63 and p.max() < 2**63
        p = p % 2**64
        return ((p >> 32) + (p % M >> 1)) % M

    s = 2 * (w + (w >> 30)) % M
    add_min = lambda x, c: np.minimum((x + c) % M, x)
    add_max = lambda x, c: np.maximum((x + c) % M, x)
    t = mul_centred((a - b) % M, s)
    assert np.array_equal(add_min(t, P), (a - b) * w % P)
    for unsigned in (False, True):
        # the same residues in the form's range: [-p, p - 1] or [1, 2p - 1]
        forms = [lambda x: x, lambda x: x - P] if not unsigned else [lambda x: np.where(x > 0, x, P), lambda x: x + P]
        for fa in forms:
            for fb in forms:
                x, y = fa(a) % M, fb(b) % M
                t = mul_centred((y - P) % M if unsigned else y, s)
                assert signed(t).min() >= -P and signed(t).max() < P
                t = add_max(t, -P)
                r = add_min(x, -P if unsigned else P)
                assert signed(t).max() < 0 and r.max() < P
                lo, hi = (r + t) % M, (r - t) % M
                assert signed(lo).min() >= -P and signed(lo).max() < P and hi.min() >= 1 and hi.max() < 2 * P
                assert np.array_equal(add_min(lo, P), (a + b * w) % P)
                assert np.array_equal(add_min(hi, -P), (a - b * w) % P)
