"""CPU test: the channel-pair layout of the transfer matrices and its multiply-accumulate.

k_mac streams, per stored row x and per pair of output channels (j, j') with
j' = Mxy j, the two complex numbers C = (A + B) / 2 and D = i (A - B) / 2 of
A = T_xj and B = conj T_xj'.  Because T_{Mxy i, Mxy j}[u] = conj T_ij[u], one
stored row feeds the inputs x and Mxy x of both channels with real operands
only (half the multiplications of the complex form).  The model below follows
k_pack (rows, columns, the second row of a row pair at the mirrored columns)
and k_mac (operands, accumulators, output) index for index, and the tests
compare it with the oracle's FP64 definition.
"""

import numpy as np
import pytest

import packed_model as M
from oracle import lf_oracle as O


class Rows:
    """Index tables of the layout (flf_api.cu build_tables)."""

    def __init__(self, N):
        self.N, self.NN, self.c = N, N * N, N // 2
        NN, c = self.NN, self.c
        self.NP = (NN + 1) // 2
        self.My = lambda i: (N - 1 - i // N) * N + i % N
        self.Mx = lambda i: (i // N) * N + (N - 1 - i % N)
        self.Tr = lambda i: (i % N) * N + i // N
        self.reps = []       # (channel, row pair?, first row)
        ops0, ops1, second = [], [], []
        mxy = lambda i: NN - 1 - i  # noqa: E731

        def generic(x):
            return (x, mxy(x), self.My(x), self.Mx(x))
        none = (-1, -1, -1, -1)

        def orbit(b, ap, trans):
            for a in (ap, N - 1 - ap):
                x = b * N + a
                self.reps.append((x, False, len(ops0)))
                ops0.append(generic(x))
                ops1.append(generic(self.Tr(x)) if trans else none)
                second.append(a > c)
        for b in range(c):
            for ap in range(b):
                orbit(b, ap, True)
        for b in range(c):
            x, y = b * N + c, self.My(b * N + c)
            X, Y = self.Tr(x), self.Tr(y)      # (c, b) and its Mx partner
            self.reps.append((x, True, len(ops0)))
            ops0 += [(x, -1, y, -1), (y, -1, x, -1)]
            ops1 += [(X, -1, -1, Y), (Y, -1, -1, X)]
            second += [False, True]
        self.nT = len(ops0)
        for b in range(c):
            orbit(b, b, False)
        x = c * N + c
        self.reps.append((x, True, len(ops0)))
        ops0 += [(x, -1, -1, -1), (-1, -1, x, -1)]
        ops1 += [none, none]
        second += [False, True]
        self.ops, self.second, self.nrow = (ops0, ops1), second, len(ops0)


def pack(Hred, N, f, t):
    """P[half block, row, pair] = (C, D)."""
    fq, NN, NP = f // 2 + 1, N * N, t.NP
    P = np.zeros((fq * fq, t.nrow, NP, 2), complex)
    for ch, pair, row in t.reps:
        spec = np.stack([np.fft.rfft2(M.kernel_image(Hred, N, ch, q, f)) for q in range(NN)]) / (f * f)
        for uy, ux, hb in M.quads(fq):
            for side, (py, px) in enumerate(((uy, ux), (ux, uy))):
                if side and uy == ux:
                    continue
                for p in range(NP):
                    j = t.Tr(p) if side else p
                    A, B = spec[j, py, px], np.conj(spec[NN - 1 - j, py, px])
                    P[hb + side, row, p] = (A + B) / 2, 1j * (A - B) / 2
                    if pair:      # the row at u*, columns mirrored
                        ps = (-py) % f
                        A, B = spec[t.My(j), ps, px], np.conj(spec[t.Mx(j), ps, px])
                        P[hb + side, row + 1, p] = (A + B) / 2, 1j * (A - B) / 2
    return P


def operands(sa, sb):
    """Real operands (p0, p1, m0, m1): P += C p0 + D p1, M += C m0 + D m1."""
    w, v = sa + np.conj(sb), sa - np.conj(sb)
    return w.real, w.imag, v.imag, -v.real


def mac(Ps, Ss, N, f, t):
    NN, NP, fq = t.NN, t.NP, f // 2 + 1
    out = np.zeros((NN, f, fq), complex)
    for uy, ux, hb in M.quads(fq):
        diag = uy == ux
        freqs = [(uy, ux), (ux, uy)]
        selfp = [(-p[0]) % f == p[0] for p in freqs]
        acc = np.zeros((2, NP, 4), complex)               # side, pair, (UP, UM, VP, VM)
        for P, S in zip(Ps, Ss):
            comb = [(S[:, p[0], p[1]], S[:, (-p[0]) % f, p[1]]) for p in freqs]
            for bs in range(1 if diag else 2):
                for r in range(t.nrow):
                    for side in range(2):
                        use = int(side != bs)
                        if use and r >= t.nT:
                            continue
                        if t.second[r] and selfp[side]:
                            continue
                        for uv in range(2):
                            a, b = t.ops[use][r][2 * uv:2 * uv + 2]
                            p0, p1, m0, m1 = operands(comb[side][uv][a] if a >= 0 else 0j, comb[side][uv][b] if b >= 0 else 0j)
                            C, D = P[hb + bs, r, :, 0], P[hb + bs, r, :, 1]
                            acc[side, :, 2 * uv] += C * p0 + D * p1
                            acc[side, :, 2 * uv + 1] += C * m0 + D * m1
        outs = np.zeros((2, 2, NN), complex)              # side, u / u*, channel
        for side in range(2):
            for p in range(NP):
                j = t.Tr(p) if side else p
                UP, UM, VP, VM = acc[side, p]
                outs[side, 0, j] = UP + 1j * UM
                outs[side, 0, NN - 1 - j] = np.conj(UP) + 1j * np.conj(UM)
                outs[side, 1, t.My(j)] = VP + 1j * VM
                outs[side, 1, t.Mx(j)] = np.conj(VP) + 1j * np.conj(VM)
        if diag:
            outs[0] += outs[1]
        for side in range(1 if diag else 2):
            py, px = freqs[side]
            if selfp[side]:
                out[:, py, px] = outs[side, 0] + outs[side, 1]
            else:
                out[:, py, px] = outs[side, 0]
                out[:, (-py) % f, px] = outs[side, 1]
    return out


@pytest.mark.parametrize("N,hs,Y,X", [(3, [7, 11], 12, 15), (5, [21, 11], 23, 17), (7, [15], 21, 28)])
def test_pair_layout_matches_oracle(N, hs, Y, X):
    rng = np.random.default_rng(N)
    nh = (N + 1) // 2
    H = [rng.random((nh, nh, h, h)) for h in hs]
    t = Rows(N)
    assert t.nrow == (t.c + 1) * (t.c + 2) and t.nT == t.c * (t.c + 1)
    f = M.choose_f(Y, X, hs, N)
    Ps = [pack(h, N, f, t) for h in H]
    vol = rng.random((len(hs), Y, X))
    fw = M.to_pixels(mac(Ps, [M.channel_spectra(v, N, f) for v in vol], N, f, t), N, f, Y, X)
    fo = O.forward_project(H, vol[:, None], N, method="direct", dtype=np.float64)[0]
    assert np.max(np.abs(fw - fo)) < 1e-12 * np.max(np.abs(fo))
    img = rng.random((Y, X))
    S = M.channel_spectra(img, N, f)
    bk = np.stack([M.to_pixels(mac([P], [S], N, f, t), N, f, Y, X) for P in Ps])
    bo = O.backward_project(H, img[None], N, method="direct", dtype=np.float64)[:, 0]
    assert np.max(np.abs(bk - bo)) < 1e-12 * np.max(np.abs(bo))
