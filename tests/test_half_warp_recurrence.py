"""CPU emulation of the half-warp permutation's partial rounds (half_partials and
its tables, p2_chain_tables, in zorch_gb300/csrc/poseidon2.cuh), word by word: lane k
holds B_k, the sum that round k will see but for the rounds in between; a round
adds j T_{k-1-r} sigma_r to it and updates each lane's own word, in runs of at most
16 rounds. The arithmetic is the kernel's (signed Montgomery words, one reduction
for four products), with every intermediate checked against the range its type and
the reduction take. Compared with the oracle's permutation for the instances in use
and for made-up ones: each of the three modes, one run, several runs and a remainder,
every exponent form."""

from __future__ import annotations

import numpy as np
import pytest

R = 1 << 32


class Words:
    """The device's arithmetic mod p on Montgomery words."""

    def __init__(self, p):
        self.p = p
        self.mu = pow(p, -1, R)  # hi - ((lo mu mod 2^32) p >> 32)

    def i32(self, x):
        assert -(1 << 31) <= x < 1 << 31
        return x

    def sredc(self, c):
        assert abs(c) <= self.p * self.p  # and so it fits 64 bits
        m = c * self.mu % R
        m = m - R if m >= R // 2 else m
        r = self.i32((c >> 32) - (m * self.p >> 32))
        assert -self.p < r < self.p and (r * R - c) % self.p == 0
        return r

    def snorm(self, x):
        assert -self.p <= x < self.p
        return x + self.p if x < 0 else x

    def word(self, x):
        assert 0 <= x < self.p
        return x

    def add(self, a, b):
        s = self.word(a) + self.word(b)
        return s - self.p if s >= self.p else s

    def sub(self, a, b):
        return self.snorm(self.word(a) - self.word(b))

    def mul(self, a, b):
        return self.snorm(self.sredc(self.word(a) * self.word(b)))

    def centred(self, x):
        return x - self.p if self.word(x) > self.p // 2 else x

    def sbox(self, x, c, alpha, factor=None):
        a = self.i32(self.word(x) + self.word(c) - self.p)
        first = a if factor is None else self.sredc(a * self.word(factor))
        a2 = self.sredc(a * a)
        if alpha == 3:
            return self.snorm(self.sredc(a2 * first))
        if alpha == 7:
            return self.snorm(self.sredc(self.sredc(a2 * first) * self.sredc(a2 * a2)))
        y, v = R % self.p, self.add(x, c)
        for _ in range(alpha):
            y = self.mul(y, v)
        return y if factor is None else self.mul(y, factor)


class Tables:
    """p2_chain_tables."""

    def __init__(self, f, diag, j, one, rp):
        runs = (rp + 15) // 16
        self.chain = (rp + runs - 1) // runs if runs else 0
        self.e = f.add(j, diag[0])
        self.mode = 0 if f.add(self.e, j) else (2 if j == one else 1)
        pw = [one] * 16
        self.m, self.t = [], []
        for _ in range(16):
            t, row = 0, [0] * 16
            for i in range(1, 16):
                t = f.add(t, pw[i])
                row[i] = f.centred(f.mul(j, pw[i]))
                pw[i] = f.mul(pw[i], diag[i])
            self.m.append(row)
            self.t.append(f.mul(j, t))


def partials(f, tab, x, rc, alpha, diag, j):
    """half_permute_a's runs over the lanes of one half-warp."""
    for r0 in range(0, len(rc), tab.chain or 1):
        n = min(tab.chain, len(rc) - r0)
        xc = [f.centred(v) for v in x]
        B = []
        for k in range(16):
            part = [f.sredc(sum(tab.m[k][i] * xc[i] for i in range(4 * g, 4 * g + 4) if i))
                    for g in range(4)]
            q = [f.snorm(v) for v in part]
            B.append(f.add(f.add(q[0], q[1]), f.add(q[2], q[3])))
        w = [0] + tab.t[:15]
        s0, b = x[0], B[0]
        for r in range(n):
            y = f.sbox(s0, rc[r0 + r], alpha, j if tab.mode == 1 else None)
            jy = y if tab.mode else f.mul(y, j)
            sigma = f.add(jy, b)
            s0 = f.sub(b, jy) if tab.mode else f.add(f.mul(y, tab.e), b)
            x = [f.add(sigma, f.mul(diag[l], x[l])) for l in range(16)]
            B = [f.add(B[k], f.mul(w[k], sigma)) for k in range(16)]
            b = B[(r + 1) & 15]
            w = [w[0]] + w[:15]  # __shfl_up by one within the half
        x = [s0] + x[1:]
    return x


def ext(f, x):
    """half_ext_linear."""
    y = []
    for l in range(16):
        a, b, c = x[l ^ 1], x[l ^ 2], x[l ^ 3]
        nxt = c if l & 1 else a
        y.append(f.add(f.add(f.add(x[l], a), f.add(b, c)), f.add(x[l], f.add(nxt, nxt))))
    return [f.add(f.add(f.add(y[l], y[l]), y[l ^ 4]), f.add(y[l ^ 8], y[l ^ 12]))
            for l in range(16)]


def permute(f, x, ei, rc, et, alpha, diag, j, one):
    tab = Tables(f, diag, j, one, len(rc))
    x = ext(f, x)
    for row in ei:
        x = ext(f, [f.sbox(x[l], row[l], alpha) for l in range(16)])
    x = partials(f, tab, x, rc, alpha, diag, j)
    for row in et:
        x = ext(f, [f.sbox(x[l], row[l], alpha) for l in range(16)])
    return x


def _made_up(field, p, alpha, rp, mode, seed):
    """Canonical constants of an instance with the given mode; the first and last
    ones at the ends of the field."""
    rng = np.random.default_rng(seed)
    draw = lambda *s: rng.integers(0, p, size=s, dtype=np.uint64).astype(np.uint32)  # noqa: E731
    ei, et, rc, dg = draw(4, 16), draw(4, 16), draw(rp), draw(16)
    ei[0], et[-1, ::2] = p - 1, 0
    j = {0: 12345, 1: p - 7, 2: 1}[mode]
    dg[0] = (p - 2 * j) % p if mode else 3
    dg[1], dg[2] = p - 1, (p + 1) // 2
    return dict(alpha=alpha, external_initial=ei, external_terminal=et, internal_rc=rc,
                internal_diag=dg, internal_j_scale=j)


CASES = ["babybear16", "koalabear16", "sp1"] + [
    (field, alpha, rp, mode) for field in (0, 1)
    for alpha, rp, mode in [(7, 13, 0), (7, 16, 1), (3, 17, 2), (3, 33, 1), (5, 1, 0), (5, 20, 1),
                            (3, 32, 0), (7, 2, 2), (3, 0, 2)]]


@pytest.mark.parametrize("case", CASES, ids=str)
def test_half_warp_partial_rounds_equal_the_oracle(orc, case):
    if case == "babybear16":
        field, p2 = 0, orc.Poseidon2.babybear16()
        ei, et, rc, dg = p2.export_canonical()
        d = dict(alpha=7, external_initial=ei, external_terminal=et, internal_rc=rc,
                 internal_diag=dg, internal_j_scale=1)
    else:
        field = 1 if isinstance(case, str) else case[0]
        p = (orc.P_BABYBEAR, orc.P_KOALABEAR)[field]
        d = (orc.load_koalabear_fixture() if case == "koalabear16" else
             orc.load_sp1_fixture() if case == "sp1" else _made_up(field, p, *case[1:], seed=3))
        p2 = orc.Poseidon2.from_canonical(
            field, d["alpha"], np.asarray(d["external_initial"]), np.asarray(d["external_terminal"]),
            np.asarray(d["internal_rc"]), np.asarray(d["internal_diag"]),
            int(d.get("internal_j_scale", 1)))
    p = (orc.P_BABYBEAR, orc.P_KOALABEAR)[field]
    f = Words(p)
    mont = lambda v: [int(x) * R % p for x in np.asarray(v).reshape(-1)]  # noqa: E731
    rows = lambda v: [mont(r) for r in np.asarray(v).reshape(-1, 16)]  # noqa: E731
    j = mont([d.get("internal_j_scale", 1)])[0]
    dg = mont(d["internal_diag"])
    if not isinstance(case, str):
        assert Tables(f, dg, j, R % p, case[2]).mode == case[3]
    rng = np.random.default_rng(11)
    states = [[0] * 16, [p - 1] * 16, [p - 1, 0] * 8, [p // 2, p // 2 + 1] * 8]
    states += [[int(v) for v in rng.integers(0, p, size=16)] for _ in range(3)]
    for x in states:
        want = [int(v) for v in p2.permute(np.asarray(x, np.uint32))]
        assert permute(f, x, rows(d["external_initial"]), mont(d["internal_rc"]),
                       rows(d["external_terminal"]), int(d["alpha"]), dg, j, R % p) == want
