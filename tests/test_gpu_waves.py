"""The warp tier's waves against the oracle: hits that leave the wave as it is and hits that drop the rest of it, chains
longer than a lane's room, and the max_entries cut-off and -R stop inside a wave, in both occurrence layouts."""
import numpy as np
import pytest

import galn_b200
import oracle
from galn_b200 import synth
from heavy_reads import READS, check, index, oracle_results, reads_of  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workload", sorted(READS))
def test_waves_against_oracle(index, workload):  # noqa: F811
    """With a normal and a small arena; the reads that outgrow the small one start anew in the team tier, and without it
    are queued for the big-arena warps."""
    ref, prefix = index
    reads, opts = reads_of(ref, workload)
    o = oracle_results(prefix, reads, opts)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=64, t0_aln=4, keep_stats=True)
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        for arena, pops in ((8192, 32768), (32, 32768), (8192, 0), (32, 0)):
            ix.set_warp_tier(True, arena)
            ix.set_team_pops(pops)
            check(galn_b200.aln(ix, opts, reads), o)
            fetch = ix.last_profile(len(reads))["fetch"].astype(np.uint64)
            np.testing.assert_array_equal(fetch, o.fetch64 if layout == 64 else o.fetch80)
            if arena == 32:
                assert (ix.last_team()["reads"] if pops else ix.last_warp_queue()["queued"]) > 0
    ix.close()


@pytest.mark.parametrize("trace", [False, True])
@pytest.mark.parametrize("n", [1, 31, 2369, 16384, 16385])
def test_job_sizes_around_the_direct_warp_tier(index, n, trace):  # noqa: F811
    """Jobs of up to 16384 reads go to the warp tier at once when it takes all of their reads (not when one is too long
    for it); larger ones through the first tier. The oracle's results either way."""
    ref, prefix = index
    ox = oracle.Index(prefix + ".bwt")
    ix = galn_b200.Index(prefix)
    ix.set_trace(trace)
    for length in (50, 300) if n <= 31 else (50,):
        r = synth.simulate_reads(ref, n, 71 + n, length, sub_rate=0.01, random_frac=0.02)
        seq, off = r.ascii(), r.off
        o = oracle.aln(ox, oracle.opt_bytes(oracle.parse_aln_args([])), oracle.encode_queries(seq, off), off,
                       np.diff(off).astype(np.int32), oracle.batches_for(n), 0)
        res = galn_b200.aln(ix, [], galn_b200.Reads(seq, off))
        np.testing.assert_array_equal(res.n_aln, o.n_aln)
        np.testing.assert_array_equal(res.pops, o.pops)
        if trace:
            np.testing.assert_array_equal(res.trace, o.trace)
        assert res.records.tobytes() == o.records.tobytes()
        prof = ix.last_profile()
        direct = n <= 16384 and length <= 256
        assert (prof["tier_reads"][0] == 0) == direct and (not direct or prof["tier_reads"][1] >= n)
    ix.close()


@pytest.mark.parametrize("opts", [[], ["-l", "10", "-k", "1"], ["-n", "3", "-M", "0", "-O", "0", "-E", "0", "-m", "500"]])
@pytest.mark.parametrize("trace", [False, True])
def test_odd_reads_take_every_route(index, opts, trace):  # noqa: F811
    """Empty and one-base reads, reads of ambiguous bases, reads past the warp tier's length, in one job: the warp tier at
    once, the persistent first tier with deep and shallow stacks, and the plain engine give the oracle's results; penalties
    of zero too."""
    ref, prefix = index
    r = synth.simulate_reads(ref, 300, 91, lambda rng, m: rng.integers(1, 120, size=m), sub_rate=0.02, random_frac=0.1)
    short = [bytes(r.ascii()[r.off[i]:r.off[i + 1]]) for i in range(300)]
    odd = [b"", b"A", b"N", b"N" * 40, b"ACGTN" * 12, short[0][:30] + b"NN" + short[1][:30]]
    long = [bytes(x) for x in np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(3).integers(0, 4, (4, 300))]]
    for reads in (short + odd, short + odd + long):
        R = galn_b200.Reads.from_strings(reads)
        o = oracle_results(prefix, R, opts)
        for setting in ("direct", 16, 1024, "plain"):
            ix = galn_b200.Index(prefix)
            ix.set_trace(trace)
            if isinstance(setting, int):
                ix.set_tuning(t0_cap=setting)
            engine = galn_b200.GALN_ENGINE_PLAIN if setting == "plain" else galn_b200.GALN_ENGINE_PERSISTENT
            check(galn_b200.aln(ix, opts, R, engine), o, trace)
            ix.close()
