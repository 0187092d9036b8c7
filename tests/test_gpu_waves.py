"""The warp tier's waves against the oracle: hits that leave the wave as it is and hits that drop the rest of it, chains
longer than a lane's room, and the max_entries cut-off and -R stop inside a wave, in both occurrence layouts."""
import numpy as np
import pytest

import galn_b200
import oracle
from galn_b200 import build, synth
import fixture_index

pytestmark = pytest.mark.gpu

READS = {
    # workload: (reads, generator arguments, options); the cut-off sets end many searches in mid-chain
    "adna": (4000, dict(length=synth.adna_lengths, sub_rate=0.005, random_frac=0.05, deaminate=0.3), synth.ADNA_OPTS),
    "divergent": (120, dict(length=100, sub_rate=0.04, indel_rate=0.005), synth.DIVERGENT_OPTS),
    "cutoff": (300, dict(length=100, sub_rate=0.04, indel_rate=0.005), synth.DIVERGENT_OPTS + ["-m", "3000"]),
    "long": (1500, dict(length=200, sub_rate=0.01, random_frac=0.05), ["-n", "6", "-o", "1", "-R", "3"]),
    "gaps": (800, dict(length=60, sub_rate=0.02, indel_rate=0.02), ["-n", "4", "-o", "3", "-e", "4", "-M", "3", "-O", "3",
                                                                    "-E", "3", "-l", "20"]),
}


@pytest.fixture(scope="module")
def index(tmp_path_factory):
    build.build()
    oracle.build()
    d = tmp_path_factory.mktemp("team")
    ref = synth.reference_genome(1_500_000, 23, n_contigs=3)
    prefix = str(d / "ref")
    fixture_index.build_from_reference(ref, prefix)
    return ref, prefix


@pytest.mark.parametrize("workload", sorted(READS))
def test_waves_against_oracle(index, workload):
    ref, prefix = index
    n, how, opts = READS[workload]
    how = dict(how)
    r = synth.simulate_reads(ref, n, 61, how.pop("length"), **how)
    reads = galn_b200.Reads(r.ascii(), r.off)
    o = oracle.aln(oracle.Index(prefix + ".bwt"), oracle.opt_bytes(oracle.parse_aln_args(opts)),
                   oracle.encode_queries(reads.seq, reads.offset), reads.offset, np.diff(reads.offset).astype(np.int32),
                   oracle.batches_for(n), 0)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=64, t0_aln=4, keep_stats=True)
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        for arena in (8192, 32):
            ix.set_warp_tier(True, arena)
            res = galn_b200.aln(ix, opts, reads)
            np.testing.assert_array_equal(res.n_aln, o.n_aln)
            np.testing.assert_array_equal(res.pops, o.pops)
            np.testing.assert_array_equal(res.rec_offset, o.rec_off)
            assert res.records.tobytes() == o.records.tobytes()
            fetch = ix.last_profile(n)["fetch"].astype(np.uint64)
            np.testing.assert_array_equal(fetch, o.fetch64 if layout == 64 else o.fetch80)
    ix.close()


@pytest.mark.parametrize("trace", [False, True])
@pytest.mark.parametrize("n", [1, 31, 2369, 16384, 16385])
def test_job_sizes_around_the_direct_warp_tier(index, n, trace):
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
def test_odd_reads_take_every_route(index, opts, trace):
    """Empty and one-base reads, reads of ambiguous bases, reads past the warp tier's length, in one job: the warp tier at
    once, the persistent first tier with deep and shallow stacks, and the plain engine agree; penalties of zero too."""
    ref, prefix = index
    r = synth.simulate_reads(ref, 300, 91, lambda rng, m: rng.integers(1, 120, size=m), sub_rate=0.02, random_frac=0.1)
    short = [bytes(r.ascii()[r.off[i]:r.off[i + 1]]) for i in range(300)]
    odd = [b"", b"A", b"N", b"N" * 40, b"ACGTN" * 12, short[0][:30] + b"NN" + short[1][:30]]
    long = [bytes(x) for x in np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(3).integers(0, 4, (4, 300))]]
    for reads in (short + odd, short + odd + long):
        R = galn_b200.Reads.from_strings(reads)
        got = []
        for setting in ("direct", 16, 1024, "plain"):
            ix = galn_b200.Index(prefix)
            ix.set_trace(trace)
            if isinstance(setting, int):
                ix.set_tuning(t0_cap=setting)
            engine = galn_b200.GALN_ENGINE_PLAIN if setting == "plain" else galn_b200.GALN_ENGINE_PERSISTENT
            res = galn_b200.aln(ix, opts, R, engine)
            got.append((res.n_aln.tolist(), res.pops.tolist(), res.records.tobytes(), res.trace.tolist() if trace else 0))
            ix.close()
        assert all(g == got[-1] for g in got[:-1])
