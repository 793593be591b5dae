"""The decision tree of the bin-tracking Ising sweep (sweep_bins_warp, csrc/engine.cu) restated on
the CPU, lane by lane, against the plain serial Wang-Landau chain: bit-sliced agreement counts,
byte-packed positions, visit counts, the order in which a chunk's slots are published and read,
rows of one and of several chunks, short blocks, whole-row wraps.  Every table position a lane
would read has to lie inside the guard bins."""
import re

import numpy as np
import pytest

from conftest import ROOT

SRC = (ROOT / "rewl_simulator_gb300" / "csrc" / "engine.cu").read_text()
GUARD = int(re.search(r"constexpr int kGuard = (\d+);", SRC).group(1))
M32 = 0xFFFFFFFF
GUARD_VALUE = (1 << 63) - 1


class Chunks:
    def __init__(self, L):
        self.n = (L + 31) // 32
        self.base, self.rem = L // self.n, L % self.n

    def len(self, c):
        return self.base + (1 if c < self.rem else 0)

    def start(self, c):
        return c * self.base + min(c, self.rem)


def node_consts(q, D):
    lvl = q.bit_length() - 1 if q else 0
    c = dict(q=q, lvl=lvl, lvla=lvl if q else 32, want=0, anc=0, mA=0, mB=0, K=0, L80=0, first=False, last=False, path=0)
    bias, prev = 0, False
    for i in range(lvl):
        node, a = q >> (lvl - i), bool((q >> (lvl - 1 - i)) & 1)
        c["anc"] |= 1 << node
        c["want"] |= a << node
        if a:
            c["mA"] |= 0xFF << (8 * i)
            bias += 2
            c["path"] |= 1 << i
        if a and prev:
            c["mB"] |= 0xFF << (8 * i)
            bias += 1
        c["K"] |= (16 - bias) << (8 * i)
        c["L80"] |= 0x80 << (8 * i)
        if i == 0:
            c["first"] = a
        prev = a
    c["last"] = prev
    if q == 0:
        c["anc"] = c["want"] = 1
    c["pbias"] = 2 + int(c["last"])
    return c


def byte(v, j):
    return (v >> (8 * j)) & 0xFF


def node_eval(c, slot, D, qs, T, wrap, lnf):
    e, x = [int(v) for v in slot[0]], [int(v) for v in slot[1]]
    if wrap:
        e[wrap[0]] += wrap[1]
    e4 = sum(e[j] << (8 * j) for j in range(min(4, D)))
    x4 = sum(x[j] << (8 * j) for j in range(min(4, D)))
    S = (((e4 & c["mA"]) + (x4 & c["mB"])) * 0x01010101 + c["K"]) & M32
    cb = 16 if c["lvl"] == 0 else byte(S, c["lvl"] - 1)
    pb = cb + e[c["lvl"]] + (x[c["lvl"]] if c["last"] else 0)
    zc = ~((S ^ (cb * 0x01010101)) + 0x7F7F7F7F) & c["L80"]
    zp = ~((S ^ ((pb * 0x01010101 - c["pbias"] * 0x01010101) & M32)) + 0x7F7F7F7F) & c["L80"]
    nC, nP = bin(zc).count("1"), bin(zp).count("1")
    return dict(rC=(cb - 16) * qs, rP=(pb - 16 - c["pbias"]) * qs, nC=nC, nP=nP, lim=T + (nC - nP) * lnf,
                x0=(x[0] - 1) * qs)


def tree_sweeps(lat, g, pos, thr, L, qs, D, lnf):
    """lat: L x L spins +-1, g: table (window bins), pos: bin, thr: threshold per attempt."""
    rc = Chunks(L)
    nb = len(g)
    G = np.concatenate([[GUARD_VALUE] * GUARD, g, [GUARD_VALUE] * GUARD]).astype(object)
    visits = [0] * (nb + 2 * GUARD)
    words = {}
    for y in range(L):
        for c in range(rc.n):
            s0 = rc.start(c)
            words[y * rc.n + c] = sum(int(lat[y, s0 + j] < 0) << j for j in range(rc.len(c)))
    lanes = [node_consts(q, D) for q in range(1 << D)]
    slots = [[[[2] * D, [1] * D] for _ in range((32 + D - 1) // D)] for _ in range(2)]
    wraps, least = rc.n == 1, (rc.base + D - 1) // D

    def write_slots(f, up_flips, c, size, frm, buf):
        au = ~(f["su"] ^ up_flips)
        t0, c0 = au ^ f["al"], au & f["al"]
        a0, a1, a2 = t0 ^ f["t1"], c0 ^ f["c1"] ^ (t0 & f["t1"]), c0 & f["c1"]
        for j in range(frm, size):
            slots[buf][j // D][0][j % D] = ((a0 >> j) & 1) + 2 * ((a1 >> j) & 1) + 4 * ((a2 >> j) & 1)
            slots[buf][j // D][1][j % D] = 1 if j == 0 and c == 0 else 2 - 2 * ((f["al"] >> j) & 1)

    def publish(y, c, buf, cprev, acc):
        up, dn = (y - 1) % L, (y + 1) % L
        cl, cr = (c - 1) % rc.n, (c + 1) % rc.n
        n, row = rc.len(c), y * rc.n
        sw, uw, dw, lw = words[row + c], words[up * rc.n + c], words[dn * rc.n + c], words[row + cl]
        rw = words[row + cr] ^ (acc if row + cr == cprev else 0)
        lb = (sw << 1) | ((lw >> (rc.len(cl) - 1)) & 1)
        rb = (sw >> 1) | ((rw & 1) << (n - 1))
        ar, ad = ~(sw ^ rb), ~(sw ^ dw)
        f = dict(sw=sw, su=sw ^ uw, al=~(sw ^ lb), t1=ar ^ ad, c1=ar & ad)
        write_slots(f, acc if up * rc.n + c == cprev else 0, c, n, 0, buf)
        return f

    def wrap_term(y):
        sw = words[y * rc.n]
        return 1 if ((sw >> (L - 1)) ^ sw) & 1 else -1

    def nodes(buf, b, A, wrap=None, row=None):
        out = []
        for c in lanes:
            k = A + c["lvl"]
            wr = (L - 1, wrap_term(row)) if row is not None and c["first"] else wrap
            out.append(node_eval(c, slots[buf][b], D, qs, int(thr[k]) if k < len(thr) else 1, wr, lnf))
        return out

    st = dict(root=pos, aprev=0, acc=0)

    def block(cur, nlev, j0, ahead):
        shift = cur[0]["x0"] if st["aprev"] else 0
        B, pos_c, pos_p = 0, [], []
        for c, v in zip(lanes, cur):
            pc = st["root"] + v["rC"] + (shift if c["first"] else 0)
            pp = st["root"] + v["rP"] + (shift if c["first"] or c["lvl"] == 0 else 0)
            assert -GUARD <= pc < nb + GUARD and -GUARD <= pp < nb + GUARD, "read outside the guard bins"
            pos_c.append(pc), pos_p.append(pp)
            bound = G[pc + GUARD] + v["lim"] + (visits[pc + GUARD] - visits[pp + GUARD]) * lnf
            if G[pp + GUARD] < bound and c["lvla"] < nlev:
                B |= 1 << c["q"]
        nxt = ahead()
        leaf, ends = None, []
        for c in lanes:
            k = c["q"]
            if ((B ^ c["want"]) & c["anc"]) == 0:
                a = (B >> k) & 1
                if c["lvla"] < nlev:
                    ends.append((c["lvl"], pos_p[k] if a else pos_c[k]))
                if c["lvl"] == D - 1 and k:
                    assert leaf is None
                    leaf = (pos_p[k] if a else pos_c[k], c["path"] | (a << (D - 1)))
        assert sorted(e[0] for e in ends) == list(range(nlev))
        for _, p in ends:
            assert 0 <= p < nb
            visits[p + GUARD] += 1
        st["root"], path = leaf
        st["acc"] |= path << j0
        st["aprev"] = (path >> (nlev - 1)) & 1
        return nxt

    planes, up_flips = publish(0, 0, 0, -1, 0), 0
    A, left, y, ci, buf = 0, len(thr), 0, 0, 0
    n = nodes(0, 0, 0, row=0 if least == 1 else None)
    while left > 0:
        size = rc.len(ci)
        nblk, cw = (size + D - 1) // D, y * rc.n + ci
        yn, cn = y, ci + 1
        if cn == rc.n:
            yn, cn = (y + 1) % L, 0
        st["acc"] = 0

        def wrap():
            return ((size - 1) % D, wrap_term(y)) if wraps and st["acc"] & 1 else None

        f, old = planes, planes["sw"]
        assert old == words[cw]
        if least >= 3:
            late = (nblk - 2) * D

            def opening():
                if nblk == 3:
                    if wraps:
                        write_slots(f, up_flips, ci, size, late, buf)
                    return nodes(buf, 1, A + D)
                m = nodes(buf, 1, A + D)
                if wraps:
                    write_slots(f, up_flips, ci, size, late, buf)
                return m

            n = block(n, D, 0, opening)
            for b in range(1, nblk - 2):
                n = block(n, D, b * D, lambda: nodes(buf, b + 1, A + (b + 1) * D))
            pub = {}

            def penultimate():
                m = nodes(buf, nblk - 1, A + (nblk - 1) * D, wrap())
                pub.update(publish(yn, cn, buf ^ 1, cw, st["acc"]))
                return m

            n = block(n, D, (nblk - 2) * D, penultimate)
            n = block(n, size - (nblk - 1) * D, (nblk - 1) * D, lambda: nodes(buf ^ 1, 0, A + size))
            planes = pub
        elif nblk == 2:
            block(n, D, 0, lambda: None)
            n = nodes(buf, 1, A + D, wrap())
            publish(yn, cn, buf ^ 1, cw, st["acc"])
            n = block(n, size - D, D, lambda: nodes(buf ^ 1, 0, A + size))
        else:
            block(n, size, 0, lambda: None)
        words[cw] = old ^ st["acc"]
        up_flips = st["acc"]
        if least < 3:
            planes = publish(yn, cn, buf ^ 1, -1, 0)
            if nblk == 1:
                n = nodes(buf ^ 1, 0, A + size, row=yn)
        left -= size
        A += size
        y, ci, buf = yn, cn, buf ^ 1
    out = np.empty((L, L), dtype=int)
    for yy in range(L):
        for x in range(L):
            c = next(c for c in range(rc.n) if rc.start(c) <= x < rc.start(c) + rc.len(c))
            out[yy, x] = -1 if (words[yy * rc.n + c] >> (x - rc.start(c))) & 1 else 1
    return out, [int(v) + k * lnf for v, k in zip(G[GUARD:GUARD + nb], visits[GUARD:GUARD + nb])], st["root"]


def serial_sweeps(lat, g, pos, thr, L, qs, lnf):
    lat, g, nb = lat.copy(), [int(v) for v in g], len(g)
    for k, T in enumerate(thr):
        y, x = divmod(k % (L * L), L)
        s = lat[y, x]
        agree = sum(int(s == v) for v in (lat[(y - 1) % L, x], lat[(y + 1) % L, x], lat[y, (x - 1) % L], lat[y, (x + 1) % L]))
        new = pos + (agree - 2) * qs
        if 0 <= new < nb and g[new] - g[pos] < int(T):
            pos = new
            lat[y, x] = -s
        g[pos] += lnf
    return lat, g, pos


@pytest.mark.parametrize("D", [5, 4, 3])
@pytest.mark.parametrize("L", [3, 4, 5, 6, 8, 9, 10, 11, 16, 20, 30, 31, 32, 33, 37, 64, 70])
def test_tree_equals_the_serial_chain(L, D):
    rng = np.random.default_rng(100 * L + D)
    for nb, qs, hot in ((3, 1, 0.5), (40, 1, 3.0), (23, -2, 1.0), (400, 2, 2.0)):
        sweeps = 3 if L < 12 else 2 if L < 32 else 1
        lat = rng.choice([-1, 1], (L, L))
        lnf = 1000
        g = rng.integers(0, 3000, nb)
        thr = np.maximum(1, (rng.exponential(hot, sweeps * L * L) * 1500).astype(np.int64))
        pos = int(rng.integers(0, nb))
        got = tree_sweeps(lat, g, pos, thr, L, qs, D, lnf)
        ref = serial_sweeps(lat, g, pos, thr, L, qs, lnf)
        np.testing.assert_array_equal(got[0], ref[0])
        assert got[1] == ref[1] and got[2] == ref[2]
