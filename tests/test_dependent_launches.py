"""Kernels that may start while the ones before them run: every pointer whose
memory such a kernel reads and a kernel of its own pass writes goes through
after_previous, which keeps its loads behind the wait.  A source check: a load
moved ahead of the wait shows on no particular run."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "core_gb300", "csrc")

# per mesh or the caller's: written before the first kernel of a pass, which is
# an ordinary launch and waits for all of it
BEFORE_THE_PASS = {"m", "geo", "len", "half_len", "w", "sp", "verts", "tiles", "seg", "qmax", "u", "xyzq", "lm", "packed",
                   "listed", "f"}
# counters and bitmaps that the kernel reaches by atomics alone or writes itself
# before its last block reads them
OWN = {"done", "next", "next_chunk", "partials", "guard_count", "n_round", "fb_count", "err", "unresolved", "split",
       "collapse"}


def kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            start = text.index("{", i)
            depth, j = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            yield m.group(1), params, text[start:j]


def test_inputs_go_through_the_wait():
    seen = 0
    for name, params, body in kernels():
        call = re.search(r"\bafter_previous\(([^)]*)\)", body)
        if not call:
            continue
        seen += 1
        waited = {a.strip() for a in call.group(1).split(",")}
        for p in re.findall(r"\*\s*(?:__restrict__)?\s*(\w+)\s*(?:,|$)", params):
            if p in waited or p in BEFORE_THE_PASS or p in OWN or (name, p) == ("k_fast_error", "out3"):  # read back
                continue
            # what is left after the stores x[...] = value
            reads = re.sub(r"(?<![\w.])%s\s*\[[^;=]*\]\s*=(?!=)" % p, "", body)
            assert not re.search(r"(?<![\w.])%s\s*\[|\*%s\b" % (p, p), reads), (name, p)
    assert seen >= 15
