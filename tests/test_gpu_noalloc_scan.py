"""cof_search_seq_noalloc at the edges of its scan (32-nt words, 1024-start
tiles, runs of tiles, the 128-window queue, 1 to 256 guides) against the
definition in numpy: windows whose PAM cells match and that differ from the
pattern in at most mm other cells.  Rows are whole numbers: exact."""
import ctypes
import random

import numpy as np
import pytest

import randgen

pytestmark = pytest.mark.gpu
COMP = str.maketrans("ACGTNRY", "TGCANYR")


def _b4(s):
    return np.array([randgen.B4[c] for c in s], dtype=np.uint8)


def _expected(seq, filt, pats, mm):
    L, g = len(filt), _b4(seq)
    if len(seq) < L:
        return []
    g = np.where(g == 15, 0, g)  # N matches nothing
    single = (g != 0) & ((g & (g - 1)) == 0)
    win = np.lib.stride_tricks.sliding_window_view(g, L)
    sng = np.lib.stride_tricks.sliding_window_view(single, L)
    rows = []
    for i, p in enumerate(pats):
        f = filt if i < len(pats) // 2 else filt.translate(COMP)[::-1]
        fb, pb = _b4(f), _b4(p)
        ok = np.ones(len(win), bool)
        for c in range(L):
            if f[c] != "N":
                ok &= sng[:, c] & ((win[:, c] & fb[c]) != 0)
        cells = [c for c in range(L) if pb[c] != 15]
        miss = sum((~(sng[:, c] & ((win[:, c] & pb[c]) != 0))).astype(int) for c in cells)
        # (the search's own count takes a genome N under any pattern cell as a
        # mismatch, the writer's recount only under a base)
        found = sum((sng[:, c] & ((win[:, c] & pb[c]) != 0)).astype(int) for c in range(L))
        for s in np.flatnonzero(ok & (miss <= mm) & (L - found <= mm)):
            rows.append((int(s), i, int(miss[s])))
    return sorted(rows)


@pytest.mark.parametrize("n,guides,pam", [
    (5, 1, "NRG"), (23, 1, "NRG"), (54, 2, "NRG"), (1023, 3, "NRG"), (1024, 3, "NRG"),
    (1046, 1, "NRG"), (1047, 17, "NRG"), (4095, 4, "NNNRRT"), (4096, 4, "NRG"), (4118, 4, "NRG"),
    (8193, 256, "NRG"), (40_001, 5, "TTTN"), (70_003, 2, "NNN")])
def test_scan_edges(cof_mod, n, guides, pam):
    import torch
    rng = random.Random(n + guides)
    seq = randgen.random_seq(rng, n, iupac_rate=0)[:n]
    user = ["".join(rng.choice("ACGT") for _ in range(20)) for _ in range(guides)]
    if pam == "TTTN":
        filt, user = "TTTN" + "N" * 20, ["NNNN" + u for u in user]
    else:
        filt, user = "N" * 20 + pam, [u + "N" * len(pam) for u in user]
    pats = user + [u.translate(COMP)[::-1] for u in user]
    mm = 11 if n < 9000 else 8  # many candidates, so that the queues fill
    want = _expected(seq, filt, pats, mm)
    nib = np.append(_b4(seq), np.zeros(n % 2, np.uint8))
    bit4 = torch.from_numpy(nib[0::2] | (nib[1::2] << 4)).cuda()
    rows = torch.zeros((len(want) + 10, 3), dtype=torch.int32, device="cuda")
    arr = (ctypes.c_char_p * len(pats))(*[p.encode() for p in pats])
    got = ctypes.c_uint32()
    rc = cof_mod.load_library().cof_search_seq_noalloc(
        bit4.data_ptr(), n, filt.encode(), arr, len(pats), mm, rows.data_ptr(), len(rows),
        ctypes.byref(got), None)
    assert rc == 0 and got.value == len(want)
    assert sorted(map(tuple, rows[:got.value].cpu().tolist())) == want
