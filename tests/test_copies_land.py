"""A kernel that brings tiles into shared memory with bulk copies leaves only
when the last of them has landed, also when a wait ran out after the last one
was issued: shared memory that a copy still writes belongs to the next block.
Checked on the sources: the wait for the ring's last copies stands under no
condition on the producer's own success.  (Kernels whose consumers issue their
own copies have no such producer.)"""

import re

import pytest

from test_launch_reads import _functions, _text


@pytest.mark.parametrize("f,kernel", [
    ("slq_kernels.cuh", "k_stream"), ("slq_kernels.cuh", "k_spmm_tc"),
    ("slq_kernels.cuh", "k_dense_tc"), ("slq_blk.cuh", "k_spmm_blk")])
def test_the_last_copies_are_waited_for(f, kernel):
    body = {n: b for n, _, b in _functions(_text(f))}[kernel]
    assert re.search(r"bulk_copy_g2s|tma_load|gather4", body)
    # waits with the flag that is never set: the bounded ones on the way out
    outs = [m.start() for m in
            re.finditer(r"mbar_wait\(&?s?full[^;]*abort_flag \+ 1\)", body)]
    assert outs
    for at in outs:
        # the conditions of the blocks that the wait stands in
        depth, i, opened = 0, at, []
        while i > 0:
            i -= 1
            if body[i] == "}":
                depth += 1
            elif body[i] == "{":
                if depth:
                    depth -= 1
                else:
                    opened.append(body[:i].rstrip().rsplit("\n", 1)[-1])
        assert not any(re.search(r"!\s*ok\b", o) for o in opened), opened
