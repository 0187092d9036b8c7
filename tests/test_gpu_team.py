"""The team tier (a block of warps per heavy read): reads handed to it as they stand after any number of pops, and
reads started anew in it, give the oracle's n_aln, pops, records and block counts, also at the max_entries cut-off
and the -R and record limits."""
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
def test_team_tier_against_oracle(index, workload):
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
    handed = 0
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        # leave at once, after a few waves, late; a tiny arena sends reads that start anew; both launch forms
        for pops, arena, fused in ((1, 8192, False), (300, 8192, True), (5000, 8192, False), (1 << 40, 32, False)):
            ix.set_tuning(t0_cap=64, t0_aln=4, keep_stats=True)
            ix.set_warp_tier(True, arena)
            ix.set_team_pops(pops)
            ix.set_fused(fused)
            res = galn_b200.aln(ix, opts, reads)
            np.testing.assert_array_equal(res.n_aln, o.n_aln)
            np.testing.assert_array_equal(res.pops, o.pops)
            np.testing.assert_array_equal(res.rec_offset, o.rec_off)
            assert res.records.tobytes() == o.records.tobytes()
            fetch = ix.last_profile(n)["fetch"].astype(np.uint64)
            np.testing.assert_array_equal(fetch, o.fetch64 if layout == 64 else o.fetch80)
            handed += ix.last_team()["reads"]
    assert handed > n // 10, "hardly a read reached the team tier"
    ix.close()


@pytest.mark.parametrize("share", [0.8, 0.93])
def test_low_complexity_reads_with_coinciding_penalties(tmp_path, share):
    """Runs of one base where every pop has children of all four bases, and the three kinds of pushes in one list: a
    share of 192 entries stages some 40,000 pushes, more than the 8192 of one warp's log (up to 16 logs, past 16 bits,
    is what a share's counts must hold)."""
    rng = np.random.default_rng(1)
    text = rng.choice(4, 1_000_000, p=[share] + [(1 - share) / 3] * 3).astype(np.uint8)
    prefix = str(tmp_path / "ref")
    galn_b200.index_text(text, prefix)
    seqs = [bytes(np.frombuffer(b"ACGT", np.uint8)[rng.choice(4, n, p=[p] + [(1 - p) / 3] * 3)])
            for n in (60, 100, 250) for p in (1.0, share) for _ in range(4)]
    reads = galn_b200.Reads.from_strings(seqs)
    opts = ["-n", "6", "-o", "3", "-e", "6", "-M", "3", "-O", "3", "-E", "3", "-l", "1024", "-i", "0", "-d", "1000000",
            "-m", "60000", "-N"]
    o = oracle.aln(oracle.Index(prefix + ".bwt"), oracle.opt_bytes(oracle.parse_aln_args(opts)),
                   oracle.encode_queries(reads.seq, reads.offset), reads.offset, np.diff(reads.offset).astype(np.int32),
                   oracle.batches_for(len(seqs)), 0)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=64, t0_aln=4)
    ix.set_team_pops(1)
    res = galn_b200.aln(ix, opts, reads)
    assert ix.last_team()["reads"] >= len(seqs) // 2
    np.testing.assert_array_equal(res.n_aln, o.n_aln)
    np.testing.assert_array_equal(res.pops, o.pops)
    assert res.records.tobytes() == o.records.tobytes()
    ix.close()


@pytest.mark.parametrize("left,extra", [(14 << 30, ["-m", str(1 << 30)]), (3 << 30, []), (3 << 29, [])])
def test_little_device_memory(index, left, extra):
    """With most of the device's memory taken: fewer teams, a smaller arena than the cut-off asks for (-m 2^30 would be
    17 GB for one team), and less space for the states of leaving reads than they need. The oracle's results."""
    torch = pytest.importorskip("torch")
    ref, prefix = index
    n, how, opts = READS["adna"]
    how = dict(how)
    r = synth.simulate_reads(ref, n, 61, how.pop("length"), **how)
    reads = galn_b200.Reads(r.ascii(), r.off)
    o = oracle.aln(oracle.Index(prefix + ".bwt"), oracle.opt_bytes(oracle.parse_aln_args(opts + extra)),
                   oracle.encode_queries(reads.seq, reads.offset), reads.offset, np.diff(reads.offset).astype(np.int32),
                   oracle.batches_for(n), 0)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=64, t0_aln=4)
    ix.set_team_pops(1)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    if free < left:
        pytest.skip("too little device memory")
    held = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        res = galn_b200.aln(ix, opts + extra, reads)
        team = ix.last_team()["reads"]
    finally:
        del held
        torch.cuda.empty_cache()
        ix.close()
    assert team > 0
    np.testing.assert_array_equal(res.n_aln, o.n_aln)
    np.testing.assert_array_equal(res.pops, o.pops)
    assert res.records.tobytes() == o.records.tobytes()


@pytest.mark.parametrize("wait_ns", [0, 20_000])
def test_lost_queue_slots(index, wait_ns):
    """The fused launch with a wait that runs out: reads that left for the team tier are also among those the host lists
    again, and are searched once."""
    ref, prefix = index
    n, how, opts = READS["adna"]
    how = dict(how)
    r = synth.simulate_reads(ref, n, 61, how.pop("length"), **how)
    reads = galn_b200.Reads(r.ascii(), r.off)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    want = galn_b200.aln(ix, opts, reads)
    ix.set_tuning(t0_cap=16, t0_aln=4)
    ix.set_team_pops(1)
    ix.set_fused(True)
    ix.set_warp_wait(wait_ns)
    res = galn_b200.aln(ix, opts, reads)
    assert ix.last_warp_queue()["gave_up"] or wait_ns
    assert n // 4 < ix.last_team()["reads"] <= n
    np.testing.assert_array_equal(res.pops, want.pops)
    assert res.records.tobytes() == want.records.tobytes()
    ix.close()
