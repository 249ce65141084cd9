"""Kernels that start as programmatic dependents run while the kernel before
them still writes (pdl_wait() orders them, include/bpf_device.cuh).  The
read-only data path (__ldg, or a `const ... __restrict__` parameter, which lets
the compiler take it) is for data that does not change while a kernel runs, so
such a kernel may read only what no kernel writes that way: observations, the
filters' tables and constants, weights of a proposal, a training set.  Checked
in the sources, since a stale value would show only now and then."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FILES = sorted(glob.glob(os.path.join(ROOT, "libbi_b200", "csrc", "*.cu*")) +
               glob.glob(os.path.join(ROOT, "include", "*.cuh")))

# names of data that no kernel of a step or of training writes while such a
# kernel runs
CONSTANT = {"y", "yf", "a.y", "filt", "sorted", "order", "prms", "blk2f", "a.blk2f",
            "a.shift", "a.scale", "a.b3", "bias"}
# load4 of train.cu reads rows of the training set
CONSTANT_IN = {"load4": {"p"}}


def _balanced(s, i, pair):
    """The index after the bracket that closes s[i]."""
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(s[i], 0)
        i += 1
        if depth == 0:
            return i


def _functions():
    """(name, is a kernel, parameters, body) of every device function."""
    out = []
    for path in FILES:
        s = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__(global|device)__", s):
            i = s.find("(", m.end())
            while i >= 0 and s[:i].rstrip().endswith("__launch_bounds__"):
                i = s.find("(", _balanced(s, i, "()"))
            if i < 0 or re.search(r"[;{}=]", s[m.end():i]):
                continue  # a variable
            name = re.search(r"(\w+)\s*$", s[:i])
            j = _balanced(s, i, "()")
            k = re.match(r"\s*(const\s*)?\{", s[j:])
            if not name or not k:
                continue  # a declaration, an operator
            b = j + k.end() - 1
            out.append((name.group(1), m.group(1) == "global", s[i + 1:j - 1], s[b:_balanced(s, b, "{}")]))
    return out


def _dependents():
    """The dependent kernels and every function they call."""
    funcs = _functions()
    by_name = {}
    for f in funcs:
        by_name.setdefault(f[0], []).append(f)
    todo = [f for f in funcs if f[1] and "pdl_wait()" in f[3]]
    seen, out = set(), []
    while todo:
        f = todo.pop()
        if (f[0], f[2]) in seen:
            continue
        seen.add((f[0], f[2]))
        out.append(f)
        for name in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", f[3])):
            todo += [g for g in by_name.get(name, []) if not g[1]]
    return out


def test_dependent_kernels_are_found():
    names = {f[0] for f in _dependents()}
    assert {"k_batch_resample", "k_systematic_coop1", "k_l96_transition", "k_l96_transition_pair", "k_pz_transition",
            "k_batch_l96_transition", "k_batch_l96_transition_pair", "k_batch_pz_transition", "k_batch_pz_guided",
            "k_pz_net", "k_l96_step", "k_train_tile", "k_reduce_adam", "k_model_transition", "load_items",
            "load_particle", "l96_pair_step", "metropolis_ancestor", "fused_systematic_ancestor"} <= names


def test_dependents_read_what_a_kernel_writes_with_plain_loads():
    bad = []
    for name, _, params, body in _dependents():
        ok = CONSTANT | CONSTANT_IN.get(name, set())
        for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
            if p not in ok:
                bad.append(f"{name}: parameter {p} is const __restrict__")
        for a in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?([\w.]+)", body):
            if a not in ok:
                bad.append(f"{name}: __ldg of {a}")
    assert not bad, "\n".join(sorted(bad))
