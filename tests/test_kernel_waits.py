"""How the kernels leave a bounded wait that ran out, read from their sources (no GPU).

A wait is per thread. Where the next instructions are collective (tensor-memory loads, barriers), lanes that
gave up one by one would leave the others at an instruction that never completes: a timeout that has to be
reported would become a kernel that never returns. So a wait either belongs to a single thread, or it is one of
the warp-uniform forms, or its result goes through ``__syncthreads_and`` before anybody acts on it; and where a
named barrier follows a wait, either the barrier carries the result (``bar_sync_and``) or nobody leaves the loop."""
import random
import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
FILES = ("attention.cu", "delta_chunk.cu", "delta_prep.cu", "delta_scan.cu", "gemm.cu", "gemm_fp8.cu")
ONE_THREAD = re.compile(r"\blane == 0|\blead\b|\br == 0|threadIdx\.x == 0")


def _text(name):
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), (SRC / name).read_text())
    return re.sub(r"/\*.*?\*/", lambda m: " " * len(m.group()), text, flags=re.S)


def per_thread_waits(text):
    """(line, statement) of every per-lane wait that a whole warp may run and act on lane by lane."""
    bad, heads, start = [], [], 0
    call = re.compile(r"\bmbar_wait(_spin|_cluster)?\(")
    for i, c in enumerate(text):
        if c in "{};":
            stmt = text[start:i]
            if call.search(stmt) and not any(ONE_THREAD.search(h) for h in heads + [stmt]):
                rest = text[i:i + 400]
                stop = re.search(r"\bbreak\b|\breturn\b", rest)
                agreed = rest.find("__syncthreads_and")
                inline = c == "{" or "break" in stmt or "return" in stmt      # acted on in the same statement
                if not inline and rest[1:].lstrip().startswith("__syncwarp();"):
                    pass                                                      # kept, not acted on: see the walks below
                elif inline or agreed < 0 or (stop and stop.start() < agreed - 6):
                    bad.append((text.count("\n", 0, i) + 1, " ".join(stmt.split())))
            if c == "{":
                heads.append(stmt)
            elif c == "}" and heads:
                heads.pop()
            start = i + 1
    return bad


@pytest.mark.parametrize("name", FILES)
def test_waits_before_collective_instructions_are_uniform(name):
    assert per_thread_waits(_text(name)) == []


def test_row_warps_that_share_a_named_barrier_leave_together():
    scan, chunk, att = _text("delta_scan.cu"), _text("delta_chunk.cu"), _text("attention.cu")
    assert "bar.sync" not in chunk
    # the walks: row warps run their loop to its end whatever a wait returned, and skip no barrier over it
    first = scan.rindex("for (int it = 0; it < N; ++it)")
    rows = scan[first:scan.index("tma_store_wait<0>();", first)]
    assert rows.count("sync_rows();") == 4 and not re.search(r"\b(break|continue|return|ok)\b|mbar_wait", rows)
    assert len(re.findall(r"if \(ok\) ok = mbar_wait_spin\(bar, parity, p\.status\);\s+__syncwarp\(\);", scan[:first])) == 1
    # attention: the only plain barriers left stand behind an agreed one, with no wait in between
    for m in re.finditer(r"\bsync_group\(\);", att):
        before = att[:m.start()]
        assert before.rfind("bar_sync_and") > before.rfind("wait_all("), att.count("\n", 0, m.start()) + 1


def test_the_reader_of_sources_sees_a_wait_that_splits_a_warp():
    text = _text("gemm.cu")
    assert "mbar_wait_warp(&tfull" in text
    assert per_thread_waits(text.replace("mbar_wait_warp(&tfull", "mbar_wait(&tfull"))


def test_split_products_read_no_row_of_a_peer_that_they_do_not_store():
    """The cluster barrier at the end of a split product is relaxed: it waits for a read of a peer's shared memory only because the
    value read is stored before it. So the reads stop at the same row as the stores."""
    text = _text("gemm.cu")
    rows = text[text.index("void split_rows("):text.index("gemm_split_kernel(")]
    read, store = rows.index("ld_cluster_f4("), rows.index("static_cast<float*>(p.C)")
    stops = [m.start() for m in re.finditer(r"if \(r0 \+ i >= hi\) break;", rows)]
    assert rows.count("ld_cluster_f4(") == 1 and len(stops) == 2 and stops[0] < read < stops[1] < store
    assert "barrier.cluster.arrive.relaxed" in text


def miscounted_blocks(text, blocks=12, schedules=200):
    """Blocks of the attention forward whose P V product is issued before all four row warps of the tile have stored P, or never,
    over random schedules of the warps and the issuer. Barriers, their indexes and parities are the source's; the scores of block j
    are there once P V of block j - 2 is issued, and a warp that has to raise its maximum may take any time over a block."""
    wait = re.search(r"mbar_wait_spin_warp\(&p_ready\[(.+?)\], (.+?), p\.status\)", text)
    arrive = re.search(r"mbar_arrive\(&p_ready\[(\w+)\]\)", text)
    sb = re.search(r"const int sb = (t \* 2 \+ \(j & 1\));\s+const uint32_t ph", text)
    assert wait and arrive and sb and re.search(r"mbar_init\(&p_ready\[\w+\], 4\)", text)
    value = lambda expr, j: eval(expr, {"t": 0, "j": j, "sb": eval(sb.group(1), {"t": 0, "j": j})})
    bad = set()
    for seed in range(schedules):
        rng = random.Random(seed)
        pending, phase, at, done = [4] * 4, [0] * 4, [0] * 4, 0
        for _ in range(200 * blocks):
            actor = rng.choice((0, 0, 0, 1, 1, 1, 2, 2, 2, 3, "issuer"))      # warp 3 is the slow one
            if done == blocks:
                break
            if actor == "issuer":
                if phase[value(wait.group(1), done)] != value(wait.group(2), done):
                    if min(at) <= done:
                        bad.add(done)
                    done += 1
            elif at[actor] < min(done + 2, blocks):
                i = value(arrive.group(1), at[actor])
                at[actor] += 1
                pending[i] -= 1
                if pending[i] == 0:
                    pending[i], phase[i] = 4, phase[i] ^ 1
        if done < blocks:
            bad.add(done)
    return bad


def test_attention_forward_counts_each_block_of_every_row_warp():
    text = _text("attention.cu")
    assert miscounted_blocks(text) == set()
    # one barrier for both score buffers: a fast warp's next block stands in for a slow warp's
    one = re.sub(r"(mbar_wait_spin_warp\(&p_ready\[).+?\], .+?,", r"\1t], j & 1,", text)
    assert miscounted_blocks(one.replace("mbar_arrive(&p_ready[sb])", "mbar_arrive(&p_ready[t])"))
