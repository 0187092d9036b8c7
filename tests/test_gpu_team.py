"""The team tier (a block of warps per heavy read): reads handed to it as they stand after any number of pops, and
reads started anew in it, give the oracle's n_aln, pops, records and block counts, also at the max_entries cut-off
and the -R and record limits, with little device memory, and for requests of several option sets served together."""
import numpy as np
import pytest

import galn_b200
import oracle
from heavy_reads import READS, check, index, oracle_results, reads_of  # noqa: F401

pytestmark = pytest.mark.gpu

# fewest reads that reach the team tier: handed over at once, after a few waves, late, and started anew from an arena of
# 32 chunks
TEAMS = {"adna": (3000, 600, 50, 100), "divergent": (100, 100, 80, 60), "cutoff": (200, 200, 80, 100),
         "long": (1000, 800, 0, 4), "gaps": (600, 500, 200, 20)}


@pytest.mark.parametrize("workload", sorted(READS))
def test_team_tier_against_oracle(index, workload):  # noqa: F811
    ref, prefix = index
    reads, opts = reads_of(ref, workload)
    n = len(reads)
    o = oracle_results(prefix, reads, opts)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    at_once, waves, late, anew = TEAMS[workload]
    for layout in (64, 80):
        ix.set_occ_layout(layout)
        for pops, arena, fused, least in ((1, 8192, False, at_once), (300, 8192, True, waves), (5000, 8192, False, late),
                                          (1 << 40, 32, False, anew), (1 << 40, 32, True, anew)):
            ix.set_tuning(t0_cap=64, t0_aln=4, keep_stats=True)
            ix.set_warp_tier(True, arena)
            ix.set_team_pops(pops)
            ix.set_fused(fused)
            check(galn_b200.aln(ix, opts, reads), o)
            fetch = ix.last_profile(n)["fetch"].astype(np.uint64)
            np.testing.assert_array_equal(fetch, o.fetch64 if layout == 64 else o.fetch80)
            assert ix.last_team()["reads"] >= least, "hardly a read reached the team tier"
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
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=64, t0_aln=4)
    ix.set_team_pops(1)
    res = galn_b200.aln(ix, opts, reads)
    assert ix.last_team()["reads"] >= len(seqs) // 2
    check(res, oracle_results(prefix, reads, opts))
    ix.close()


def test_more_records_than_a_team_keeps(tmp_path):
    """A read with more than 4096 records goes on from the team tier to the thread tiers."""
    rng = np.random.default_rng(1)
    base = [0.8] + [0.2 / 3] * 3
    prefix = str(tmp_path / "ref")
    galn_b200.index_text(rng.choice(4, 1_000_000, p=base).astype(np.uint8), prefix)
    reads = galn_b200.Reads.from_strings([b"A" * 20] + [bytes(np.frombuffer(b"ACGT", np.uint8)[rng.choice(4, 20, p=base)])
                                                        for _ in range(16)])
    opts = ["-n", "5", "-o", "1", "-e", "2", "-l", "1024", "-N", "-R", "1000000", "-m", "60000"]
    o = oracle_results(prefix, reads, opts)
    assert 4096 < o.n_aln.max() < 30_000
    for pops in (1, 1000):
        ix = galn_b200.Index(prefix)
        ix.set_trace(False)
        ix.set_tuning(t0_cap=64, t0_aln=4)
        ix.set_team_pops(pops)
        check(galn_b200.aln(ix, opts, reads), o)
        assert ix.last_team()["reads"] > 4 and ix.last_profile()["tier_reads"][2] >= (o.n_aln > 4096).sum()
        ix.close()


@pytest.mark.parametrize("left,extra", [(14 << 30, ["-m", str(1 << 30)]), (3 << 30, []), (3 << 29, [])])
def test_little_device_memory(index, left, extra):  # noqa: F811
    """With most of the device's memory taken: fewer teams, a smaller arena than the cut-off asks for (-m 2^30 would be
    17 GB for one team), and less space for the states of leaving reads than they need. The oracle's results."""
    torch = pytest.importorskip("torch")
    ref, prefix = index
    reads, opts = reads_of(ref, "adna")
    o = oracle_results(prefix, reads, opts + extra)
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
    check(res, o)


@pytest.mark.parametrize("wait_ns", [0, 20_000])
def test_lost_queue_slots(index, wait_ns):  # noqa: F811
    """The fused launch with a wait that runs out: reads that left for the team tier are also among those the host lists
    again, and are searched once."""
    ref, prefix = index
    reads, opts = reads_of(ref, "adna")
    n = len(reads)
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_tuning(t0_cap=16, t0_aln=4)
    ix.set_team_pops(1)
    ix.set_fused(True)
    ix.set_warp_wait(wait_ns)
    res = galn_b200.aln(ix, opts, reads)
    assert ix.last_warp_queue()["gave_up"] or wait_ns
    assert n // 4 < ix.last_team()["reads"] <= n
    check(res, oracle_results(prefix, reads, opts))
    ix.close()


def test_requests_of_several_option_sets(index):  # noqa: F811
    """Requests with different options in one step of a server, whose reads leave the warp tier after 100 pops."""
    ref, prefix = index
    work = ["adna", "divergent", "gaps", "long"]
    parts = [reads_of(ref, w) for w in work]
    want = [oracle_results(prefix, r, opts) for r, opts in parts]
    ix = galn_b200.Index(prefix)
    ix.set_trace(False)
    ix.set_team_pops(100)
    server = galn_b200.Server(ix)
    for _ in range(2):
        ids = [server.submit(galn_b200.parse_options(opts), reads) for reads, opts in parts]
        for i, o in zip(ids, want):
            check(server.wait(i), o)
    server.close()
    ix.close()
