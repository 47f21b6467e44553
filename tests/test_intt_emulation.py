"""CPU emulation of what the inverse transform adds to the LDE's passes
(zorch_gb300/csrc/zc_ntt.cu): the message read at -i mod k in 32-bit index
arithmetic (p1_pass<REV>, lde_small_body with rev), no scaling at coset 1, the
output scale carried by pass 2's running factors (p2_first), and a row's last pass
without products for twiddle 1 (dif_group<LAST>). Restated with canonical values
over every work item of small shapes: the transform of the oracle's evaluations is
the message again, each word is read once and written once, and the butterflies
left without a product are those whose twiddle is 1."""

from __future__ import annotations

import numpy as np
import pytest
from test_ntt_fused_emulation import P, brev, pad, passes, root, row_stride

U32 = (1 << 32) - 1


def dif_group(v, tw, off, ls, sh0, r_, last, count):
    for r in range(r_):
        hb, sh = r_ - 1 - r, sh0 + r
        for j in range(1 << r_):
            if j & (1 << hb):
                continue
            j2, jm = j | (1 << hb), j & ((1 << hb) - 1)
            w = tw[(off << sh) + jm * (1 << (ls + sh))]
            u, t = v[j], v[j2]
            v[j] = (u + t) % P
            if last and jm == 0:
                assert off == 0 and ls == 0 and w == 1
                v[j2] = (u - t) % P
                count["skipped"] += 1
            else:
                v[j2] = (u - t) * w % P
                count["products"] += 1


def pass1(x, z, c, tile, lk1, lk2, lti, max_r, reads, count):
    """lde_pass1_fused<REV> at h = 1, one coset: unit, so nothing is scaled."""
    k2, ti, lk = 1 << lk2, 1 << lti, lk1 + lk2
    rs, ps, kmask = row_stride(k2), passes(lk2, max_r), (1 << lk) - 1
    work = [None] * (ti * rs)
    tw = [pow(root(lk2), i, P) for i in range(max(k2 // 2, 1))]
    i1_0 = tile * ti
    zd = (c << lk) + i1_0
    for q, (h0, r_) in enumerate(ps):
        first, last, ls = q == 0, q == len(ps) - 1, h0 - r_ + 1
        for it in range(1 << (lti + lk2 - r_)):
            d, g = it & (ti - 1), it >> lti
            off, blk = g & ((1 << ls) - 1), g >> ls
            base = (blk << (h0 + 1)) | off
            ar = d * rs + pad(base)
            if first:
                i0 = (i1_0 + d + (off << lk1)) & U32
                v = []
                for j in range(1 << r_):
                    i = (0 - i0 - (j << (ls + lk1))) & U32 & kmask
                    assert i == -(i1_0 + d + ((off + (j << ls)) << lk1)) % (1 << lk)
                    reads[(c, i)] = reads.get((c, i), 0) + 1
                    v.append(x[(c << lk) + i])
            else:
                v = [work[ar + pad(j << ls)] for j in range(1 << r_)]
            dif_group(v, tw, 0 if last else off, 0 if last else ls, lk2 - 1 - h0, r_, last, count)
            for j in range(1 << r_):
                if last:
                    z[zd + d + (brev(base, lk2) << lk1) + (brev(j, r_) << (lk1 + lk2 - r_))] = v[j]
                else:
                    work[ar + pad(j << ls)] = v[j]


def passes2(lk1, max_r):
    """Pass 2's: the smaller radix first where a warp would span two rows."""
    ps = passes(lk1, max_r)
    if len(ps) > 1 and lk1 - ps[0][1] < 5:
        r0 = lk1 // len(ps)
        ps = [(lk1 - 1, r0)] + passes(lk1 - r0, max_r)
    return ps


def pass2(z, out, c, tile, lk1, lk2, ltt, max_r, post, writes, count):
    """lde_pass2_fused at blowup 1, natural order, outputs scaled by post."""
    k1, lk = 1 << lk1, lk1 + lk2
    rs, wk = row_stride(k1), root(lk)
    work = [None] * ((1 << ltt) * rs)
    tw = [pow(root(lk1), i, P) for i in range(max(k1 // 2, 1))]
    ps = passes2(lk1, max_r)

    def put(pos, val):
        out[pos] = val
        writes[pos] = writes.get(pos, 0) + 1

    for q, (h0, r_) in enumerate(ps):
        first, last, ls = q == 0, q == len(ps) - 1, h0 - r_ + 1
        for it in range(1 << (ltt + lk1 - r_)):
            if first:
                off, dt = it & ((1 << ls) - 1), it >> ls
                t = (tile << ltt) + dt
                f = pow(wk, t * off & ((1 << lk) - 1), P) * post % P
                step = pow(wk, (t << ls) & ((1 << lk) - 1), P)
                src = (c << lk) + (t << lk1) + off
                v = []
                for j in range(1 << r_):
                    v.append(z[src + (j << ls)] * f % P)
                    f = f * step % P
                base, ar = off, dt * rs + pad(off)
            else:
                dt, g = it & ((1 << ltt) - 1), it >> ltt
                t = (tile << ltt) + dt
                off, blk = g & ((1 << ls) - 1), g >> ls
                base = (blk << (h0 + 1)) | off
                ar = dt * rs + pad(base)
                v = [work[ar + pad(j << ls)] for j in range(1 << r_)]
            dif_group(v, tw, 0 if last else off, 0 if last else ls, lk1 - 1 - h0, r_, last, count)
            for j in range(1 << r_):
                if last:
                    put((c << lk) + t + (brev(base + j, lk1) << lk2), v[j])
                else:
                    work[ar + pad(j << ls)] = v[j]


def _evaluations(orc, lk, cols, seed):
    """Random messages and their evaluations by the oracle's transform."""
    x = np.random.default_rng(seed).integers(0, P, size=(cols, 1 << lk)).astype(np.uint32)
    y = orc.from_mont(0, orc.rs_encode(0, orc.to_mont(0, x), 0))
    return x, [int(v) for v in np.asarray(y).reshape(-1)]


SHAPES = [  # log_k1, log_k2, log_ti, log_tt, largest radix
    (4, 4, 2, 1, 4),   # one pass a row
    (4, 3, 4, 0, 4),   # k1 != k2, a tile of the whole row
    (5, 4, 3, 2, 2),   # three passes and two
    (6, 6, 3, 3, 4),
    (7, 6, 4, 3, 3),   # first, middle and last
    (5, 5, 2, 1, 5),   # radix 2^5
    (6, 7, 1, 4, 5),
]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_four_step_inverse(orc, shape):
    lk1, lk2, lti, ltt, max_r = shape
    lk, cols = lk1 + lk2, 2
    x, y = _evaluations(orc, lk, cols, lk)
    z, out = [None] * len(y), [None] * len(y)
    reads, writes = {}, {}
    c1, c2 = {"skipped": 0, "products": 0}, {"skipped": 0, "products": 0}
    for c in range(cols):
        for tile in range(1 << (lk1 - lti)):
            pass1(y, z, c, tile, lk1, lk2, lti, max_r, reads, c1)
    assert len(reads) == len(y) and set(reads.values()) == {1} and None not in z
    post = pow((P + 1) // 2, lk, P)
    for c in range(cols):
        for tile in range(1 << (lk2 - ltt)):
            pass2(z, out, c, tile, lk1, lk2, ltt, max_r, post, writes, c2)
    assert len(writes) == len(y) and set(writes.values()) == {1}
    assert out == [int(v) for v in x.reshape(-1)]
    # all butterflies, and those of the last pass at twiddle 1
    for count, lm, ps in ((c1, lk2, passes(lk2, max_r)), (c2, lk1, passes2(lk1, max_r))):
        assert count["skipped"] + count["products"] == cols * (1 << (lk - 1)) * lm
        r = ps[-1][1]
        assert count["skipped"] == cols * (1 << (lk - r)) * ((1 << r) - 1)


@pytest.mark.parametrize("lk", [0, 1, 2, 5, 7])
def test_single_pass_inverse(orc, lk):
    """lde_small_body with rev and post, one coset at shift 1."""
    k, cols = 1 << lk, 3
    x, y = _evaluations(orc, lk, cols, 50 + lk)
    post, rs = pow((P + 1) // 2, lk, P), row_stride(k)
    tw = [pow(root(lk), i, P) for i in range(max(k // 2, 1))]
    for c in range(cols):
        work = [None] * rs
        for idx in range(k):
            work[pad(idx & (k - 1))] = y[(c << lk) + ((-idx & U32) & (k - 1))] * post % P
        count = {"skipped": 0, "products": 0}
        for h0, r_ in passes(lk, 4):
            ls = h0 - r_ + 1
            for g in range(1 << (lk - r_)):
                off, blk = g & ((1 << ls) - 1), g >> ls
                ar = pad((blk << (h0 + 1)) | off)
                v = [work[ar + pad(j << ls)] for j in range(1 << r_)]
                dif_group(v, tw, off, ls, lk - 1 - h0, r_, ls == 0, count)
                for j in range(1 << r_):
                    work[ar + pad(j << ls)] = v[j]
        assert [work[pad(brev(t, lk))] for t in range(k)] == [int(v) for v in x[c]]
