"""`galn index` on the GPU: all five files equal to the reference builder's for every golden FASTA (the
library call and the command line), the .bwt/.sa of random, repetitive and tiny texts equal to the
oracle's, a larger genome-like reference equal to the fixture builder's (pinned itself to the reference),
and an index the builder wrote searched to the reference's .sai bytes."""
import filecmp
import os
import subprocess
import threading

import numpy as np
import pytest

import galn_b200
import oracle
from conftest import GOLDEN, case_paths, golden_cases
import fixture_index as index_build
from galn_b200 import build, synth

pytestmark = pytest.mark.gpu
INDEX_CASES = sorted(os.listdir(os.path.join(GOLDEN, "index")))
EXTS = ("pac", "ann", "amb", "bwt", "sa")


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    oracle.build()


def _fasta(d):
    gz = os.path.join(d, "ref.fa.gz")
    return gz if os.path.exists(gz) else os.path.join(d, "ref.fa")


def _same(a, b):
    return filecmp.cmp(a, b, shallow=False)


@pytest.mark.parametrize("d", [os.path.join(GOLDEN, "index", c) for c in INDEX_CASES] +
                         [os.path.join(GOLDEN, "small"), os.path.join(GOLDEN, "genome")])
def test_golden_fasta(d, tmp_path):
    pre = str(tmp_path / "g")
    st = galn_b200.index_fasta(_fasta(d), pre)
    for ext in EXTS:
        assert _same(pre + "." + ext, os.path.join(d, "ref." + ext)), ext
    assert st["n"] == 2 * len(oracle.forward_from_pac(pre + ".pac"))
    assert st["sort_passes"] >= 8 and st["ms_device"] > 0


def test_command_line(tmp_path):
    d = os.path.join(GOLDEN, "index", "repeats")
    pre = str(tmp_path / "c")
    p = subprocess.run([build.CLI, "index", "-v", "-p", pre, _fasta(d)], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    for ext in EXTS:
        assert _same(pre + "." + ext, os.path.join(d, "ref." + ext)), ext
    p = subprocess.run([build.CLI, "index", "-a", "cpu", "-p", pre, _fasta(d)], capture_output=True, text=True)
    assert p.returncode == 1


def _texts():
    rng = np.random.default_rng(77)
    yield "random", rng.integers(0, 4, 250_000)
    yield "homopolymer", np.zeros(6000, np.int64)
    yield "dinucleotide", np.tile([0, 1], 4000)
    yield "period7", np.tile(rng.integers(0, 4, 7), 2000)
    u = rng.integers(0, 4, 20_000)
    yield "repeats", np.concatenate([u, rng.integers(0, 4, 100), u, 3 - u[::-1], u[:5000]])
    yield "palindrome", np.concatenate([u[:8000], 3 - u[:8000][::-1]])
    for n in (1, 2, 3, 4, 5, 15, 16, 17, 63, 64, 65, 127, 128, 129, 2047, 2048, 2049, 4095, 4096, 4097):
        yield f"len{n}", rng.integers(0, 4, n)


@pytest.mark.parametrize("name,F", list(_texts()), ids=[t[0] for t in _texts()])
def test_texts_against_oracle(name, F, tmp_path):
    F = np.asarray(F, dtype=np.uint8)
    galn_b200.index_text(F, str(tmp_path / "g"))
    oracle.index_files(F, str(tmp_path / "o"))
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("g." + ext)), str(tmp_path / ("o." + ext))), ext


# suffixes the 64-bit path sorts at once, per text: small enough for several buckets and round chunks where
# the text allows it (a homopolymer's suffixes share one prefix and one group, so it needs the whole text)
WIDE_CHUNK = {"random": 31_250, "repeats": 16_000, "palindrome": 4_000}


@pytest.mark.parametrize("name,F", list(_texts()), ids=[t[0] for t in _texts()])
def test_texts_64bit_path_against_oracle(name, F, tmp_path):
    """The builder's 64-bit path (bucketed first sort, doubling rounds in chunks of whole groups, BWT and
    samples scattered from the ranks) forced on the same texts: the oracle's .bwt and .sa."""
    F = np.asarray(F, dtype=np.uint8)
    chunk = WIDE_CHUNK.get(name, 2 * len(F))
    st = galn_b200.index_text(F, str(tmp_path / "w"), sort_chunk=chunk)
    oracle.index_files(F, str(tmp_path / "o"))
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("w." + ext)), str(tmp_path / ("o." + ext))), ext
    assert st["n"] == 2 * len(F)


def test_genome_shape_64bit_path_equals_32bit_path(tmp_path):
    """8 Mbp with repeat families, tandem repeats and N runs (16 M suffixes): the 64-bit path with a million
    suffixes per sort (many buckets, many chunks per round) writes the 32-bit path's files."""
    ref = synth.reference_genome(8_000_000, 31, n_contigs=5)
    fa = str(tmp_path / "ref.fa")
    synth.write_fasta(fa, ref)
    galn_b200.index_fasta(fa, str(tmp_path / "n"))
    F = oracle.forward_from_pac(str(tmp_path / "n.pac"))
    st = galn_b200.index_text(F, str(tmp_path / "w"), sort_chunk=1 << 20)
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("w." + ext)), str(tmp_path / ("n." + ext))), ext
    assert st["rounds"] >= 2 and st["sorted_items"] > st["n"]


def test_genome_shape_against_fixture_builder(tmp_path):
    """8 Mbp with repeat families, tandem repeats and N runs: the fixture builder (prefix doubling on
    torch.sort, byte-identical to the reference builder on the golden genomes) gives the same five files."""
    ref = synth.reference_genome(8_000_000, 31, n_contigs=5)
    fa = str(tmp_path / "ref.fa")
    synth.write_fasta(fa, ref)
    index_build.build_index(fa, str(tmp_path / "fx"))
    st = galn_b200.index_fasta(fa, str(tmp_path / "gp"))
    for ext in EXTS:
        assert _same(str(tmp_path / ("gp." + ext)), str(tmp_path / ("fx." + ext))), ext
    assert st["rounds"] >= 2


def test_search_on_a_built_index(tmp_path):
    """The aDNA golden case searched on the index this builder wrote gives the reference's .sai bytes."""
    pre = str(tmp_path / "s")
    galn_b200.index_fasta(os.path.join(GOLDEN, "small", "ref.fa"), pre)
    meta = golden_cases()["adna"]
    p = case_paths("adna", meta)
    res = galn_b200.aln(galn_b200.Index(pre), meta["opts"], p["fq"])
    assert res.sai_bytes() == open(p["sai"], "rb").read()


@pytest.mark.parametrize("n,at", [(1, 0), (40, 39), (5000, 17)])
@pytest.mark.parametrize("sort_chunk", [0, 256])
def test_code_above_3_is_refused(tmp_path, n, at, sort_chunk):
    """A sequence with a code other than 0..3 is refused by both paths, and nothing is written."""
    f = np.random.default_rng(n).integers(0, 4, n).astype(np.uint8)
    f[at] = 4
    with pytest.raises(galn_b200.GalnError):
        galn_b200.index_text(f, str(tmp_path / "x"), sort_chunk=sort_chunk)
    assert not os.listdir(tmp_path)


@pytest.mark.parametrize("symbols", [16, 32])
@pytest.mark.parametrize("name,F", list(_texts()), ids=[t[0] for t in _texts()])
def test_texts_with_both_first_round_keys(name, F, symbols, tmp_path):
    """The 32-bit path with 16-symbol 32-bit keys (texts of 2^24 symbols and more) and with 32-symbol 64-bit keys
    (shorter ones) forced on the same texts: the oracle's .bwt and .sa."""
    F = np.asarray(F, dtype=np.uint8)
    galn_b200.index_text(F, str(tmp_path / "g"), first_symbols=symbols)
    oracle.index_files(F, str(tmp_path / "o"))
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("g." + ext)), str(tmp_path / ("o." + ext))), ext


@pytest.mark.parametrize("d", [os.path.join(GOLDEN, "index", c) for c in INDEX_CASES] +
                         [os.path.join(GOLDEN, "small"), os.path.join(GOLDEN, "genome")])
def test_golden_texts_with_16_symbol_keys(d, tmp_path):
    F = oracle.forward_from_pac(os.path.join(d, "ref.pac"))
    galn_b200.index_text(F, str(tmp_path / "g"), first_symbols=16)
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("g." + ext)), os.path.join(d, "ref." + ext)), ext


@pytest.mark.parametrize("bp,passes", [((1 << 23) - 1, 8), (1 << 23, 4)])
def test_lengths_around_the_change_of_keys(bp, passes, tmp_path):
    """2^24 - 2 and 2^24 suffixes of a genome-like text, on both sides of the line between the two kinds of keys (8 and
    4 passes in the first round): the 64-bit path's files."""
    ref = synth.reference_genome(9_000_000, 31, n_contigs=5)
    fa = str(tmp_path / "ref.fa")
    synth.write_fasta(fa, ref)
    galn_b200.fasta_to_pac(fa, str(tmp_path / "p"))
    F = oracle.forward_from_pac(str(tmp_path / "p.pac"))[:bp].copy()
    st = galn_b200.index_text(F, str(tmp_path / "g"))
    assert st["n"] == 2 * bp and st["rounds"] >= 1
    later = (st["n"].bit_length() + (st["n"] - 1).bit_length() + 7) // 8          # passes over a later round's rank pairs
    assert st["scatter_items"] - st["n"] * passes == later * (st["sorted_items"] - st["n"])
    galn_b200.index_text(F, str(tmp_path / "w"), sort_chunk=1 << 20)
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("g." + ext)), str(tmp_path / ("w." + ext))), ext


def test_genome_shape_with_16_symbol_keys_against_fixture_builder(tmp_path):
    """9 Mbp (18 M suffixes, above the line) with repeat families, tandem repeats and N runs: the fixture builder's five
    files."""
    ref = synth.reference_genome(9_000_000, 33, n_contigs=5)
    fa = str(tmp_path / "ref.fa")
    synth.write_fasta(fa, ref)
    index_build.build_index(fa, str(tmp_path / "fx"))
    st = galn_b200.index_fasta(fa, str(tmp_path / "gp"))
    for ext in EXTS:
        assert _same(str(tmp_path / ("gp." + ext)), str(tmp_path / ("fx." + ext))), ext
    assert st["n"] >= 1 << 24 and st["rounds"] >= 2


@pytest.mark.parametrize("symbols", [16, 32])
@pytest.mark.parametrize("tail", ["A", "AAAAAAAAAAAAAAAA", "CAAAAAAAAAAAAAA", "TTTTTTTTTTTTTTT"])
def test_text_ends_inside_a_first_round_key(tmp_path, tail, symbols):
    """Texts that start and end with runs (the text ends with the reverse complement of its start): suffixes shorter than
    the first round's keys, of 16 or 32 symbols, stand before longer ones with the same key, as the 64-bit path's keys
    have it."""
    code = {"A": 0, "C": 1, "G": 2, "T": 3}
    rng = np.random.default_rng(5)
    run = np.array([code[c] for c in tail], np.uint8)
    f = np.concatenate([3 - run[::-1], rng.integers(0, 4, 3000).astype(np.uint8), run, run])
    for name, how in (("a", dict(first_symbols=symbols)), ("b", dict(sort_chunk=700))):
        galn_b200.index_text(f, str(tmp_path / name), **how)
    for ext in (".bwt", ".sa"):
        assert open(str(tmp_path / ("a" + ext)), "rb").read() == open(str(tmp_path / ("b" + ext)), "rb").read()


@pytest.mark.parametrize("name,F", [t for t in _texts() if t[0] in ("random", "repeats", "period7", "len1", "len4097")])
def test_block_that_cannot_be_had(name, F, tmp_path):
    """A text whose one block of device memory cannot be allocated is built by the 64-bit path, not refused."""
    F = np.asarray(F, dtype=np.uint8)
    galn_b200.index_text(F, str(tmp_path / "g"), max_block=1)
    oracle.index_files(F, str(tmp_path / "o"))
    for ext in ("bwt", "sa"):
        assert _same(str(tmp_path / ("g." + ext)), str(tmp_path / ("o." + ext))), ext


@pytest.mark.parametrize("n", [3000, 9_000_000])
def test_files_through_pipes(n, tmp_path):
    """.bwt and .sa written to named pipes, read one after the other: the bytes of the files, small and large."""
    F = np.random.default_rng(n).integers(0, 4, n).astype(np.uint8)
    galn_b200.index_text(F, str(tmp_path / "f"))
    got = []
    for ext in (".bwt", ".sa"):
        os.mkfifo(str(tmp_path / ("p" + ext)))
    reader = threading.Thread(target=lambda: got.extend(open(str(tmp_path / ("p" + ext)), "rb").read()
                                                        for ext in (".bwt", ".sa")), daemon=True)
    reader.start()
    galn_b200.index_text(F, str(tmp_path / "p"))
    reader.join(30)
    assert got == [open(str(tmp_path / ("f" + ext)), "rb").read() for ext in (".bwt", ".sa")]
