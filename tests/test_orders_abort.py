"""Who may act on the order kernel's abort flag (csrc/orders.cu).

Any role raises the flag when a bounded wait runs out, so two warps that read it for
themselves can see different values, and lanes of one warp can too.  Where they then
part before a named barrier (bar.sync has no bound) or a full-mask warp barrier, the
CTA waits forever.  A hang cannot be tested on the GPU; the rule that excludes it can
be read off the source: the scan warps, which meet at named barriers, take thread 0's
reading, published before the barrier that ends an order, and a warp of another role
decides by vote."""
import os
import re

import ocrt_gb300

SRC = os.path.join(os.path.dirname(ocrt_gb300.__file__), "csrc", "orders.cu")


def _roles():
    text = open(SRC).read()
    body = text[text.index("orders_body("):text.index("#define OR_ARGS")]
    body = re.sub(r"//[^\n]*", "", body.replace("// =====", "@@"))
    parts = [p.split("\n", 1)[1] for p in body.split("@@")[1:]]
    assert len(parts) == 3, "scan warps, producers, MMA issue"
    return parts


def _reads(part):
    """Statements that read the flag (stores to it left out)."""
    out = []
    for line in part.split("\n"):
        code = re.sub(r"\*b\.abort = 1;", "", line)
        if "b.abort" in code and "or_wait" not in code:
            out.append(code.strip())
    return out


def test_scan_warps_take_one_reading():
    scan, _, _ = _roles()
    reads = _reads(scan)
    assert reads
    for r in reads:
        assert r.startswith("if (tid == 0)"), r
    # published before the barrier that ends an order, acted on after it; two slots, as
    # the next order's reading may be stored while a slow warp still looks at this one
    end = scan.index("quit[ph & 1] = *b.abort")
    bar = scan.index("or_bar(1, 256);", end)
    step = scan.index("++ph;", bar)
    assert scan.index("quit[(ph & 1) ^ 1]) break;", step) > step
    assert scan.count("quit[") == 2


def test_other_warps_vote():
    _, producers, issue = _roles()
    issue = issue[:issue.index("umma_commit(b.fin)")]          # past it all threads meet at the CTA's barrier
    for part in (producers, issue):
        reads = _reads(part)
        assert reads
        for r in reads:
            assert "__any_sync(0xffffffffu, *b.abort != 0)" in r, r
