"""Kernels launched by programmatic dependent launch (pdl.cuh) may be resident
while the kernel before them still runs.  The read-only loads that the compiler
forms by itself (__ldg, const __restrict__ parameters) may be moved above the
wait for it, so those kernels read by load_ro, which stays behind it, and only
what no kernel ahead writes while they live, or by plain loads; the constant
lists of a plan may be read anyhow."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "topopt3d_b200", "csrc")


def balanced(s, i, pair):
    """End of the bracketed text that opens at s[i]."""
    depth = 0
    for j in range(i, len(s)):
        depth += {pair[0]: 1, pair[1]: -1}.get(s[j], 0)
        if depth == 0:
            return j
    raise ValueError("unbalanced source")


def functions(src):
    """name -> (qualifier, parameters, body) of the device functions of a
    file, comments removed."""
    src = re.sub(r"//[^\n]*", "", src)
    out = {}
    for m in re.finditer(r"__(global|device)__", src):
        head = re.compile(r"\b(\w+)\s*\(").search(src, m.end())
        while head and head.group(1) in ("__launch_bounds__", "sizeof"):
            end = balanced(src, head.end() - 1, "()")
            head = re.compile(r"\b(\w+)\s*\(").search(src, end)
        if not head:
            continue
        end = balanced(src, head.end() - 1, "()")
        brace = src.find("{", end)
        if brace < 0 or src[end + 1:brace].strip() not in ("", "const"):
            continue
        out.setdefault(head.group(1), []).append(
            (m.group(1), src[head.end():end], src[brace:balanced(src, brace, "{}")]))
    return out


def dependent_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = open(path).read()
        names = set(re.findall(r"\blaunch_pdl\(\s*(k_\w+)", src))
        for n in sorted(names):
            yield pytest.param(path, n, id=f"{os.path.basename(path)}:{n}")


def read_only(params, body):
    """What of a function uses the read-only path."""
    bad = re.findall(r"__ldg\s*\([^;]*", body)
    for p in params.split(","):
        if "__restrict__" in p and re.search(r"\bconst\b", p.split("*")[0]) and not re.search(
                r"\bint[24]?\s*\*", p):
            bad.append(p.strip())
    return bad


@pytest.mark.parametrize("path,name", list(dependent_kernels()))
def test_operands_of_a_dependent_launch_stay_behind_the_wait(path, name):
    fns = functions(open(path).read())
    assert name in fns
    bad, seen, todo = [], set(), [name]
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for _, params, body in fns[f]:
            bad += [(f, b) for b in read_only(params, body)]
            todo += [g for g in fns if g not in seen and re.search(rf"\b{g}\b", body)]
    assert not bad
    body = fns[name][0][2]
    assert "pdl_wait()" in body


@pytest.mark.parametrize("path,name", [p for p in dependent_kernels() if "coarse_inv" not in p.id])
def test_dependents_are_released_after_the_last_store(path, name):
    """What a dependent reads by load_ro is not written while it lives: the
    release comes after the kernel's stores, and after its wait.  (The kernels
    of the coarsest inverse release before them and read by plain loads.)"""
    body = functions(open(path).read())[name][0][2]
    release = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
    stores = [m.start() for m in re.finditer(r"\]\s*[+\-*]?=\s|\bsym_out_v\b", body)]
    assert len(release) == 1
    assert release[0] > max(stores) and release[0] > body.index("pdl_wait()")


def test_the_coarsest_inverse_reads_by_plain_loads():
    src = open(os.path.join(CSRC, "kernels_coarse_inv.cu")).read()
    assert "load_ro" not in src
