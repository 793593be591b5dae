"""How far the nodes of a block of the global-table kernel's tree (sweep_tables_warp, csrc/engine.cu) can lie
from the bin it starts in: the kernel's bound, taken from its source, against every path through the last block
of random Ashkin-Teller rows.  A node beyond the bound would be looked up in another bin's slot of the cache."""
import re
from itertools import product
from types import SimpleNamespace

import numpy as np
import pytest

from conftest import ROOT

SRC = (ROOT / "rewl_simulator_gb300" / "csrc" / "engine.cu").read_text()
FAR = re.search(r"^ +far = (.*);", SRC, re.M).group(1)
REACH = re.search(r"const int reach = TREE \? (.*) \* \(int\)__reduce_max_sync\(kFull, \(unsigned\)far\) : 0;", SRC).group(1)
D = 5
UNIT = 1 << 20


def _rows(L, K, sigma_h, bin_width, n, seed):
    """Position changes of n random rows' flips in plane a, as the kernel forms them for a row that is one chunk:
    of each site, of each after its left neighbour has flipped less that, of the last after the first has flipped
    less that; and the binary places below a bin."""
    r = np.random.default_rng(seed)
    a, b = r.choice([-1, 1], (2, n, 3, L)).astype(np.int64)
    h = np.round(r.normal(0, sigma_h, (n, L)) * UNIT).astype(np.int64)
    J, K = UNIT, int(round(K * UNIT))
    if np.log2(bin_width) % 1 == 0:
        mul, sh = 1, 20 + int(np.log2(bin_width))
    else:
        mul, sh = int(round(1 / bin_width)), 20
    zm = min((mul & -mul).bit_length() - 1, sh)
    even = 1 if zm < sh else 0
    shz, mulz = sh - zm - even, mul >> zm
    J, K, h = J * mulz, K * mulz, h * mulz
    ai, bi = a[:, 1], b[:, 1]
    left, right = np.roll(ai, 1, 1), np.roll(ai, -1, 1)
    bl, br = np.roll(bi, 1, 1), np.roll(bi, -1, 1)
    sa = a[:, 0] + left + right + a[:, 2]
    sab = a[:, 0] * b[:, 0] + left * bl + right * br + a[:, 2] * b[:, 2]
    d = 2 * ai * (h * bi + J * sa + K * bi * sab) >> even
    dl = -4 * ai * left * (J + K * bi * bl) >> even
    dl[:, 0] = 0
    wrap = -4 * ai[:, -1] * right[:, -1] * (J + K * bi[:, -1] * br[:, -1]) >> even
    return d, dl, wrap, shz


def _bound(d, dl, wrap, shz):
    """The kernel's reach of each row, by its own expressions."""
    far = []
    for lane in range(d.shape[1]):
        last = np.abs(wrap) if lane == d.shape[1] - 1 else 0 * wrap
        ns = dict(max=np.maximum, abs=np.abs, shz=shz, last=last, d=SimpleNamespace(x=d[:, lane], y=dl[:, lane]))
        far.append(eval(FAR, {"__builtins__": {}}, ns))
    return eval(REACH, {"__builtins__": {}}, {"D": D}) * np.max(far, axis=0)


def _farthest(d, dl, wrap, shz):
    """The farthest bin from the block's first one that a node of the row's last block names."""
    n, L = d.shape
    j0 = (L - 1) // D * D
    out = np.zeros(n, dtype=np.int64)
    for path in product((0, 1), repeat=L - j0):
        for before, head in product((0, 1), (0, 1) if j0 else (path[0],)):
            pos, prev = np.zeros(n, dtype=np.int64), before if j0 else 0
            for k, taken in enumerate(path):
                j = j0 + k
                to = pos + d[:, j] + prev * dl[:, j] + (head * wrap if j == L - 1 else 0)
                for start in (0, (1 << shz) - 1):                  # positions within the block's first bin
                    out = np.maximum(out, np.abs(start + to >> shz))
                if taken:
                    pos = to
                prev = taken
    return out


@pytest.mark.parametrize("L", range(3, 13))
@pytest.mark.parametrize("K, sigma_h, bin_width", [(0.75, 0.5, 0.05), (1.0, 0.0, 0.05), (0.95, 1.0, 0.05), (-0.9, 0.7, 0.05),
                                                   (0.5, 0.5, 0.25), (1.0, 2.0, 1.0), (0.0, 0.5, 0.05)])
def test_no_node_lies_beyond_the_reach(L, K, sigma_h, bin_width):
    rows = _rows(L, K, sigma_h, bin_width, 20000, 17 * L)
    assert np.all(_farthest(*rows) <= _bound(*rows))
