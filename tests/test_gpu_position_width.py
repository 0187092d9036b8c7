"""The search with 32-bit BWT positions (texts shorter than 2^32 - 64 symbols) and with 64-bit ones, on both
sides of that line: the longest text of the one and the shortest of the other, whose rows reach the last values
32 bits hold and, in the 80-symbol layout, a second superblock. Pseudo-random symbols in BWA's .bwt layout
(tests/bwt_synth.py); n_aln, pops, traces and records equal the oracle's, with trace hashes on and, off, through the
first tier, the warp tier and the team tier."""
import numpy as np
import pytest

import bwt_synth
import galn_b200
import oracle
from galn_b200 import build

pytestmark = pytest.mark.gpu
NARROW = (1 << 32) - 64
COMP = np.array([3, 2, 1, 0], np.uint8)


def _spelled_reads(words, ox, rows, primary, length):
    """Reads that the index holds: the reverse complements of the `length` symbols before each row's suffix."""
    hdr, body = words[:10].view(np.uint64), words[10:]
    C = np.array([0, hdr[1], hdr[2], hdr[3]], np.uint64)
    sym = np.zeros((len(rows), length), np.uint8)
    ok = np.ones(len(rows), bool)
    for t in range(length):
        ok &= rows != primary
        r = np.where(rows == primary, 0, rows).astype(np.uint64)
        p = r - (r > primary)
        w = body[(p >> 7) * 16 + 8 + ((p & 127) >> 4)]
        c = ((w >> (30 - 2 * (p & 15)).astype(np.uint32)) & 3).astype(np.uint8)
        sym[:, length - 1 - t] = c
        rows = C[c] + ox.occ4(r)[np.arange(len(rows)), c]
    return np.frombuffer(b"ACGT", np.uint8)[COMP[sym[ok][:, ::-1]]]


@pytest.mark.parametrize("n", [NARROW - 1, NARROW])
def test_positions_on_both_sides_of_the_line(n):
    build.build()
    oracle.build()
    primary, length = n - 12_345, 40
    words = bwt_synth.random_bwt(n, primary, seed=7)
    ox = oracle.Index(file_words=words)
    ix = galn_b200.Index(bwt_bytes=words)
    ix.set_tuning(t0_cap=256)            # reads cross into the warp tier too
    rng = np.random.default_rng(3)
    top = np.arange(n - 400, n + 1, dtype=np.uint64)      # rows at the top of the range
    rows = np.concatenate([top, rng.integers(0, n + 1, size=600, dtype=np.uint64)])
    rand = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=(300, length))]
    seq = np.concatenate([_spelled_reads(words, ox, rows, primary, length), rand]).copy()
    m = len(seq)
    off = np.arange(m + 1, dtype=np.int64) * length
    opts = ["-n", "4", "-l", "1024"]
    query = oracle.encode_queries(seq.reshape(-1), off)
    o = oracle.aln(ox, oracle.opt_bytes(oracle.parse_aln_args(opts)), query, off, np.full(m, length, np.int32),
                   oracle.batches_for(m))
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        res = galn_b200.aln(ix, opts, galn_b200.Reads(seq.reshape(-1), off))
        np.testing.assert_array_equal(res.n_aln, o.n_aln)
        np.testing.assert_array_equal(res.pops, o.pops)
        np.testing.assert_array_equal(res.trace, o.trace)
        np.testing.assert_array_equal(res.records, o.records)
    assert (res.records["k"] >= (1 << 31)).any() and (res.n_aln > 0).mean() > 0.5
    ix.set_trace(False)
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        # most reads in the first tier; all in the warp tier; states handed to the team tier after a wave and after
        # several, by both launch forms; and reads that start anew there (the random ones outgrow a small arena)
        for cap, pops, arena, fused, teams in ((4096, 0, 8192, False, 0), (16, 0, 8192, False, 0), (16, 1, 8192, False, 1200),
                                               (16, 1, 8192, True, 1200), (16, 200, 8192, False, 250),
                                               (16, 1 << 40, 32, False, 250)):
            ix.set_tuning(t0_cap=cap, t0_aln=4, keep_stats=True)
            ix.set_warp_tier(True, arena)
            ix.set_team_pops(pops)
            ix.set_fused(fused)
            res = galn_b200.aln(ix, opts, galn_b200.Reads(seq.reshape(-1), off))
            np.testing.assert_array_equal(res.n_aln, o.n_aln)
            np.testing.assert_array_equal(res.pops, o.pops)
            np.testing.assert_array_equal(res.records, o.records)
            fetch = ix.last_profile(m)["fetch"].astype(np.uint64)
            np.testing.assert_array_equal(fetch, o.fetch64 if layout == 64 else o.fetch80)
            assert ix.last_team()["reads"] >= teams
    ix.close()
