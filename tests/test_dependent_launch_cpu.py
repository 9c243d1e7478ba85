"""Kernels that start before their predecessor has ended (programmatic dependent launch), read as
source.

A read-only load (ld.global.nc: what the compiler may make of a const __restrict__ pointer) needs data
that nothing writes while the kernel runs, and such a kernel runs before griddepcontrol.wait returns.
So whatever an earlier kernel of an iteration writes (vectors, scalars, flags) comes in by plain
pointers; matrices, index lists and other data of the set-up or the assembly may be read-only.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "waterscapes_gb300", "csrc")
FILES = ("solve.cu", "patch.cuh", "tile.cuh")

# data of the mesh, the set-up, the assembly or the start of a solve
STATIC = {"rp", "ci", "va", "skl", "soff", "sci", "sva", "dg", "sl", "perm", "cols", "vals", "inc_ptr", "inc",
          "cell_nodes", "cdat", "node_bc", "tab", "dinv", "cinv", "vinst", "Q", "lo", "len", "inst", "cptr", "chunks",
          "target", "sh_node", "sh_ptr", "node_inst", "tiles"}


def _source(name):
    s = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", s)


def _match(s, i, a, b):
    """Index past the bracket that closes s[i] == a."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == a) - (s[k] == b)
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced")


def _functions(s):
    """(name, parameters, body) of every device function and kernel definition."""
    for m in re.finditer(r"__(?:global|device)__", s):
        p = m.end()
        lb = re.match(r"\s*(?:__forceinline__\s*)?(?:void\s*)?__launch_bounds__\s*\(", s[p:])
        if lb:
            p = _match(s, p + lb.end() - 1, "(", ")")
        h = re.match(r"[\s\w*<>:,&]*?\b(\w+)\s*\(", s[p:])
        if not h:
            continue
        e = _match(s, p + h.end() - 1, "(", ")")
        b = re.match(r"\s*\{", s[e:])
        if b:
            yield h.group(1), s[p + h.end():e - 1], s[e:_match(s, e + b.end() - 1, "{", "}")]


def _all():
    return [f for name in FILES for f in _functions(_source(name))]


def test_the_reader_finds_the_kernels():
    names = {n for n, _, _ in _all()}
    assert {"k_spmv", "spmv_sell_body", "k_spmv_tile", "k_patch_sys", "k_mr_dot", "k_bmr_beta"} <= names


def test_every_kernel_launched_dependent_waits_for_its_predecessor():
    text = "".join(_source(n) for n in FILES)
    launched = set(re.findall(r"launch_k\(c,\s*(k_\w+)", text)) | set(re.findall(r"auto kern = (k_\w+)", text))
    waits = {n: "pdl_wait()" in b or "spmv_sell_body" in b for n, _, b in _all()}
    launched.discard("k_spmv_staged")  # an ordinary launch
    assert launched and all(waits[n] for n in launched)


def test_what_earlier_kernels_write_is_not_read_only():
    bad = []
    for name, par, body in _all():
        if "pdl_wait()" not in body and "spmv_sell_body" not in body and name not in ("slice_frozen", "patch_robin"):
            continue
        for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s*(\w+)", par):
            if p not in STATIC:
                bad.append((name, p))
    assert not bad
