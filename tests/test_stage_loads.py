"""The kernels that come up while the one in front still runs (stage_begin and
launch_next) must read its results with ordinary loads: the read-only path
(__ldg, or a const __restrict__ pointer that the compiler may send there) is
defined only for memory that nothing writes while the grid lives."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rforest_b200",
                   "csrc", "kernels.cu")
# every device function through which those kernels reach residues or records
READERS = ["contract_terms", "contract_tiles", "load_points", "inv_run", "crt_coeff", "crt_range",
           "crt_dispatch", "k_contract", "k_inv_team", "k_inv_cta", "k_crt_mixed", "k_crt_finish"]


def _function(text, name):
    """Parameters and body of the device function or kernel `name`."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        rest = text[i:].lstrip()
        if not rest.startswith("{"):
            continue  # a call
        j = start = text.index("{", i)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                return text[m.end():i], text[start:j]
    raise AssertionError("no definition of %s" % name)


def test_every_early_kernel_is_listed():
    text = open(SRC).read()
    early = set(re.findall(r"launch_next\(\s*(k_\w+)", text))
    assert early and early <= set(READERS)
    for name in early:
        assert re.match(r"\{\s*stage_begin\(\);", _function(text, name)[1]), name


def test_results_of_the_kernel_in_front_are_not_read_as_constant():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    for name in READERS:
        params, body = _function(text, name)
        assert "__ldg" not in body, name
        for decl in re.findall(r"const\s+(?:uint32_t|CrtRec)\s*\*\s*__restrict__\s+(\w+)",
                               params + body):
            assert decl == "idx", "%s: %s" % (name, decl)  # (uploaded before, by a copy)
