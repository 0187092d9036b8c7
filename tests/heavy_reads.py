"""Reads whose searches are long, of several kinds, on one genome with repeats, and what the oracle says of them: shared by
the tests of the warp and team tiers."""
import numpy as np
import pytest

import galn_b200
import oracle
from galn_b200 import build, synth
import fixture_index

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


def reads_of(ref, workload):
    """The workload's reads and options."""
    n, how, opts = READS[workload]
    how = dict(how)
    r = synth.simulate_reads(ref, n, 61, how.pop("length"), **how)
    return galn_b200.Reads(r.ascii(), r.off), opts


def oracle_results(prefix, reads, opts):
    return oracle.aln(oracle.Index(prefix + ".bwt"), oracle.opt_bytes(oracle.parse_aln_args(opts)),
                      oracle.encode_queries(reads.seq, reads.offset), reads.offset, np.diff(reads.offset).astype(np.int32),
                      oracle.batches_for(len(reads)), 0)


def check(res, o, trace=False):
    np.testing.assert_array_equal(res.n_aln, o.n_aln)
    np.testing.assert_array_equal(res.pops, o.pops)
    if trace:
        np.testing.assert_array_equal(res.trace, o.trace)
    np.testing.assert_array_equal(res.rec_offset, o.rec_off)
    assert res.records.tobytes() == o.records.tobytes()
