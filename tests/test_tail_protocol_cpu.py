"""The words that the blocks of the tail launch leave for one another, checked on
the CPU over every order in which a few blocks can get on, with the sizes the
kernel is compiled with."""
import functools
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@functools.lru_cache(None)
def compiled(expr: str) -> str:
    """An expression over the device descriptors, evaluated by a host program."""
    import tempfile
    from kgmt_gb300.build import nvcc
    include = Path(nvcc()).resolve().parent.parent / "include"
    with tempfile.TemporaryDirectory() as d:
        src, exe = Path(d) / "t.cpp", Path(d) / "t"
        src.write_text(f'#include <cuda_runtime.h>\n#include <iostream>\n#include <type_traits>\n#include "kgmt_types.h"\n'
                       f"using namespace kgmt;\nint main() {{ std::cout << ({expr}); }}\n")
        subprocess.run(["g++", "-std=c++17", f"-I{include}", f"-I{ROOT / 'kgmt_gb300' / 'csrc'}", str(src), "-o", str(exe)], check=True)
        return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


def stale_reads(blocks: int, meetings: int, rows: int) -> set:
    """(meeting, meeting whose word was read) of every read that is not of the
    reader's own meeting.  A block writes its word, arrives, waits for all
    arrivals, reads every word, and goes on; meeting m uses row m % rows."""
    start = tuple((0, 0) for _ in range(blocks)), tuple((-1,) * blocks for _ in range(rows))
    todo, seen, bad = [start], {start}, set()
    while todo:
        at, words = todo.pop()
        for b, (m, step) in enumerate(at):
            if m == meetings:
                continue
            new_words = words
            if step == 0:  # write
                row = list(words[m % rows])
                row[b] = m
                new_words = words[:m % rows] + (tuple(row),) + words[m % rows + 1:]
            elif step == 1:  # arrive: counted below by how far each block is
                pass
            elif step == 2:  # wait
                if any((mm, ss) < (m, 2) for mm, ss in at):
                    continue
            else:
                got = words[m % rows][step - 3]
                if got != m:
                    bad.add((m, got))
            nxt = (m, step + 1) if step < 2 + blocks else (m + 1, 0)
            s = at[:b] + (nxt,) + at[b + 1:], new_words
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return bad


@pytest.mark.parametrize("blocks", [2, 3])
def test_meeting_words_are_read_before_they_are_written_again(blocks):
    rows = int(compiled("sizeof(TailScratch::word) / (sizeof(uint32_t) * kTailMaxBlocks)"))
    assert stale_reads(blocks, 3, rows) == set()


def test_one_row_of_words_would_not_do():
    assert (0, 1) in stale_reads(2, 2, 1)


def test_appended_rows_are_compared_with_the_accepted_samples():
    """Two counts of the same samples, made apart (one before the rows are placed,
    one while they are), in the tail launch as in the chain's finaliser: a
    difference is reported.  Nothing a caller passes makes them differ, so that
    each compares them is read from the source."""
    csrc = ROOT / "kgmt_gb300" / "csrc"
    for name, start in (("kgmt_iter.cuh", "void finalize_query("), ("kgmt_tail.cuh", "k_tail(const QueryParams*")):
        body = (csrc / name).read_text().split(start, 1)[1]
        body = body[:body.index("\n}\n")]
        line = [l for l in body.splitlines() if "kErrAppendMismatch" in l]
        assert len(line) == 1 and "!=" in line[0] and "atomicOr(&sched->error" in line[0], name


def test_score_flags_hold_whole_tags():
    """A flag may be left from any earlier launch of the engine, so the tag of an
    iteration (launch number << 17, plus the iteration) must not come round: 2^40
    launches are thousands of years of planning."""
    flag = "std::remove_reference_t<decltype(TailScratch::scored[0])>"
    for launches in (1, 1 << 11, 1 << 15, 1 << 40):
        assert compiled(f"({flag}(({launches}ull + 7) << 17)) != ({flag}(7ull << 17))") == "1", launches


def node_share(trees, blocks=152) -> int:
    """The old nodes a block takes of the query with the most a block, divided as
    the launch divides them (float32)."""
    f = np.float32
    n = np.array(trees, np.uint64)
    weight = (n + np.uint64(31)) >> np.uint64(5)
    if len(n) == 1:
        nb = np.array([blocks])
    else:
        nb = 1 + (f(blocks - len(n)) * f(0.99999) * (weight.astype(f) * (f(1) / f(weight.sum())))).astype(np.int64)
    share = (n.astype(f) * f(1.00001) * (f(1) / nb.astype(f))).astype(np.int64) + 1
    return int(((share + 3) & ~3).max())


def test_counts_fit_the_exchanged_word():
    """A block's word has as many bits for its re-activated nodes as an iteration
    that the launch takes can need: all old nodes of the block (a large epsilon
    re-activates every node).  Trees that a card holds can have more."""
    nodes, bits = int(compiled("kTailNodes")), int(compiled("kExchangeBits - kRepeatBits"))
    assert nodes < 1 << bits
    assert node_share([1 << 28]) <= nodes < node_share([17_000_000] * 32)
    body = (ROOT / "kgmt_gb300" / "csrc" / "kgmt_tail.cuh").read_text()
    assert "share > (warp == 0 ? kTailShare : kTailNodes)" in body and "if(s_too_large | s_too_many)" in body
