"""Kernels that are launched before the launch that writes their input has ended (programmatic
dependent launch) must not read it through the read-only path, and not before they have waited.
Read from the sources: nothing of it shows in results until a line is stale."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "su2_b200", "csrc")
# read-only while a chain runs: a batch's tile tables, buffer indices and trajectory number,
# which change between the chains only
TABLES = {"ch", "of", "cur", "traj"}


def strip_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def closing(text, i, pair):
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k
    raise AssertionError("unbalanced")


def kernels(path):
    """(name, parameters, body) of every __global__ function of a source file."""
    text = strip_comments(open(path).read())
    for m in re.finditer(r"__global__\s+void", text):
        i = m.end()
        b = re.compile(r"\s*__launch_bounds__\s*").match(text, i)
        if b:
            i = closing(text, b.end(), "()") + 1
        name = re.compile(r"\s*(\w+)\s*\(").match(text, i)
        end = closing(text, name.end() - 1, "()")
        brace = text.index("{", end)
        yield name.group(1), text[name.end():end], text[brace:closing(text, brace, "{}") + 1]


def chained():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        out += [(os.path.basename(path), *k) for k in kernels(path)
                if re.search(r"\bpdl_(start|wait)\b", k[2])]
    return out


CHAINED = chained()


def test_the_chained_kernels_are_found():
    names = {k[1] for k in CHAINED}
    assert {"k_force_su2", "k_force_su2_link", "k_force_su2_planes", "k_force_su2_split",
            "k_force_su2_xsplit", "k_force_su2_pair", "k_plaq_accept_su2", "k_force_vjp",
            "k_force_vjp_gather", "k_batch_force", "k_batch_plaq", "k_batch_reduce_accept",
            "k_metro_su2", "k_metro_su2_wide"} <= names
    launched = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        launched |= set(re.findall(r"launch_force\(\s*(k_\w+)",
                                   strip_comments(open(path).read())))
    assert launched <= names, launched - names


@pytest.mark.parametrize("src,name,params,body", CHAINED, ids=[f"{k[0]}-{k[1]}" for k in CHAINED])
def test_chained_kernel_reads_its_input_coherently(src, name, params, body):
    read_only = re.findall(r"const\s+[\w:<>]+\s*\*\s*__restrict__\s+(\w+)", params)
    assert set(read_only) <= TABLES, f"{src}: {name} takes {read_only} for the read-only path"
    # __ldg of the tables alone
    assert not [a for a in re.findall(r"__ldg\(([^)]*)\)", body) if a != "&of[tile]"]
    # FP64 links are read below the wait only if their addresses come out of it
    waits = re.findall(r"pdl_(?:start|wait)(?:<.*?>)?\(([^()]*)\);", body)
    own_loads = "ld_link" in body or re.search(r"\b(force_\w+_impl|force_half_x|staple_pair|"
                                               r"plaq_site|plaq_bands|pair_link|vjp_site)\b",
                                               body)
    assert waits
    if own_loads and "ld_link_rw" not in body:
        assert all(waits), f"{src}: {name} waits without the index of its loads"


def test_shared_loads_take_the_ordinary_path():
    """The loads that the chained kernels share, and the bodies they call."""
    common = strip_comments(open(os.path.join(CSRC, "su2b_common.cuh")).read())
    for m in re.finditer(r"ld_link(?:_rw)?\(const Link(?:32|64) \*p\) \{", common):
        body = common[m.end():closing(common, m.end() - 1, "{}")]
        assert ".nc" not in body and "__ldg" not in body
    ops = strip_comments(open(os.path.join(CSRC, "site_ops.cuh")).read())
    assert ".nc" not in ops and "__ldg" not in ops
    for f in ("adjoint.cu", "gauge.cu", "metropolis.cu"):
        text = strip_comments(open(os.path.join(CSRC, f)).read())
        assert ".nc." not in text and "__ldg" not in text, f
    pairs = strip_comments(open(os.path.join(CSRC, "pairs.cu")).read())
    i = pairs.index("ld_pair(")
    assert "__ldg" not in pairs[i:closing(pairs, pairs.index("{", i), "{}")]
