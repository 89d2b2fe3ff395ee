"""The one-pass form of the wide kernel writes to the reductions' scratch arrays itself in places. A reduction (bu::...) leads with a barrier, but its
result is read from the scratch after its last one: what a warp writes there next must have a barrier, or another reduction, in between, on every
way through the code. Checked on the source, block by block."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gorch_b200", "csrc")
READS = {"sum_d3": {"d0", "d1", "u"}, "sum_d": {"d0"}, "sum_i": {"i0"}, "min_i2": {"i0", "i1"}, "min_i": {"i0"}, "max_i": {"i0"}, "max_u3": {"i0", "i1", "u"},
         "max_u64": {"u"}, "min_u64": {"u"}, "scan_excl_d2": {"d0", "d1"}, "scan_excl_d": {"d0"}}
TOKEN = re.compile(r"(?P<sync>__syncthreads\s*\()|bu::(?P<red>\w+)\s*<|(?P<alias>\w+)\s*=\s*reinterpret_cast<\w+\*>\((?:sh\.)?sc\.(?P<of>\w+)\)"
                   r"|(?P<write>\b(?:sh\.)?(?:sc\.)?\w+)\[[^\]=]*\]\s*=(?!=)|(?P<open>\{)|(?P<close>\})|(?P<els>\belse\b)|(?P<cond>\bif\b)")


def unsafe_writes(src):
    """Writes to an array that a warp may still be reading a reduction's result from: (offset, array)."""
    src = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), src)
    found, alias = [], {}
    busy, stack = set(), []                    # arrays still being read; per open block: (state before it, state after the `then` of its if)
    last_if, pending_else = False, None
    for m in TOKEN.finditer(src):
        kind = m.lastgroup if m.lastgroup != "of" else "alias"
        if kind == "sync":
            busy = set()
        elif kind == "red":
            busy = set(READS.get(m["red"], ()))
        elif kind == "alias":
            alias[m["alias"]] = m["of"]
        elif kind == "write":
            name = m["write"].split(".")[-1]
            arr = alias.get(name) if "sc." not in m["write"] else name
            if arr in busy:
                found.append((m.start(), arr))
        elif kind == "open":
            stack.append((set(busy), last_if, pending_else))
            pending_else = None
        elif kind == "close" and stack:
            before, was_if, other = stack.pop()
            if other is not None:              # end of an else: either branch
                busy = busy | other
            elif was_if:
                if re.match(r"\s*else\b", src[m.end():]):
                    pending_else, busy = busy, before
                else:
                    busy = busy | before
        last_if = kind == "cond" or (last_if and kind not in ("open", "close"))
    return found


@pytest.mark.parametrize("name", ["sample_wide_onepass.cuh", "sample_wide.cuh"])
def test_no_write_while_a_result_is_read(name):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    assert "bu::" in src
    bad = [(src.count("\n", 0, at) + 1, arr) for at, arr in unsafe_writes(src)]
    assert bad == []


def test_the_check_sees_both_branches():
    body = "float* w = reinterpret_cast<float*>(sc.d0); if (low) { x = bu::sum_d<8>(x, sc, tid); } else { __syncthreads(); } w[warp] = 1;"
    assert unsafe_writes(body) and not unsafe_writes(body.replace("w[warp]", "__syncthreads(); w[warp]"))
