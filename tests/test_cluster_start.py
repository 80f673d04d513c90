"""Blocks of a cluster reach into each other's shared memory only once all of
them run: CUDA asks for a cluster barrier between a kernel's start and its first
access to another block's shared memory.  Nothing on the GPU shows its absence
reliably, so the order is read from the sources: in every kernel that maps
another block's shared memory, itself or in a function that it calls, a cluster
barrier comes first."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cctag_b200" / "csrc"

REMOTE = r"\bmap_shared_rank\s*\("
BARRIER = r"\bthis_cluster\s*\(\s*\)\s*\.\s*(?:sync|barrier_wait)\s*\("


def functions(text):
    """(header, name, body) of every function definition in CUDA source text."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    out = []
    for m in re.finditer(r"__(?:global|device)__[^;{}]*?\b(\w+)\s*\((?:[^(){};]|\([^(){};]*\))*\)\s*(?:const\s*)?\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += (text[i] == "{") - (text[i] == "}")
            i += 1
        out.append((m.group(0), m.group(1), text[m.end():i - 1]))
    return out


def remote_accessors(funcs):
    """Names of the device functions that map another block's shared memory, or call one that does."""
    names = {n for _, n, body in funcs if re.search(REMOTE, body)}
    while True:
        more = {n for _, n, body in funcs if any(re.search(rf"\b{k}\s*(?:<[^;()]*>)?\s*\(", body) for k in names)}
        if more <= names:
            return names
        names |= more


def unordered(text):
    """The kernels of the text whose first remote access no cluster barrier precedes."""
    funcs = functions(text)
    names = remote_accessors(funcs)
    bad = []
    for header, name, body in funcs:
        if "__global__" not in header or name not in names:
            continue
        access = re.compile("|".join([REMOTE] + [rf"\b{k}\s*(?:<[^;()]*>)?\s*\(" for k in names - {name}]))
        first = access.search(body).start()
        if not re.search(BARRIER, body[:first]):
            bad.append(name)
    return bad


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_remote_shared_memory_follows_a_cluster_barrier(path):
    assert unordered(path.read_text()) == []


def test_the_reading_of_the_sources_tells_the_orders_apart():
    put = "__device__ void put(int* p) { *cg::this_cluster().map_shared_rank(p, 1) = 0; }\n"
    kernel = "template <bool C> __global__ void __maxnreg__(72) k(int n) {{ __shared__ int s; {} }}"
    late = "put(&s); cg::this_cluster().sync();"
    loop = "for (int i = 0; i < n; ++i) { put(&s); cg::this_cluster().sync(); }"
    good = "if constexpr (C) cg::this_cluster().sync(); for (int i = 0; i < n; ++i) { put(&s); }"
    split = "cg::this_cluster().barrier_arrive(); s = 0; cg::this_cluster().barrier_wait(); put(&s);"
    none = "s = n;"
    got = [unordered(put + kernel.format(b)) for b in (late, loop, good, split, none)]
    assert got == [["k"], ["k"], [], [], []]


def test_the_clustered_identification_is_read():
    funcs = functions((CSRC / "identify.cu").read_text())
    assert {"k_identify", "sample_round", "gn_refine"} <= remote_accessors(funcs)
