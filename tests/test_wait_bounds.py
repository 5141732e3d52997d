"""Every bounded device-side wait records its timeout in the status word: a wait that
ran out without it would let a call return success with unfinished data.  Read from
the sources, since a wait cannot be made to run out from outside: each comparison
of elapsed time with a bound is followed, in its own block, by kDevTimeout."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avocado-sandwich_gb300", "csrc")
ELAPSED = re.compile(r"(clock64\(\)|gtimer\(\)|global_ns\(\)) - t0\)? > ")


def waits():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            lines = open(os.path.join(CSRC, name)).read().split("\n")
            for i, line in enumerate(lines):
                if ELAPSED.search(line):
                    depth, block = 0, []
                    for follow in lines[i:i + 12]:
                        block.append(follow)
                        depth += follow.count("{") - follow.count("}")
                        if depth <= 0:
                            break
                    yield "%s:%d" % (name, i + 1), "\n".join(block)


def test_every_wait_that_runs_out_records_it():
    found = list(waits())
    assert len(found) >= 6
    silent = [where for where, block in found if "kDevTimeout" not in block]
    assert silent == []
