"""Kernels launched in a chain (``chained`` in csrc/common.cuh): what the launch accepts, and the rule that every such kernel waits
for the one before it.  No GPU: the first compiles, the second reads the sources."""
import os
import re
import subprocess

import pytest

from qutai_b200 import build

LAUNCHES = """
#include <type_traits>
#include "common.cuh"
using namespace qmoe;
__global__ void kernel(const float* in, __nv_bfloat16* out, long long n, int m) {}
template <typename... A, typename = decltype(chained(kernel, 1, 32, 0, nullptr, std::declval<A>()...))>
std::true_type accepted(int);
template <typename... A>
std::false_type accepted(...);
template <typename... A>
constexpr bool takes = decltype(accepted<A...>(0))::value;
static_assert(takes<const float*, __nv_bfloat16*, long long, int>, "the kernel's own types");
static_assert(takes<float*, __nv_bfloat16*, int, long long>, "conversions that any call makes");
static_assert(!takes<__nv_bfloat16*, float*, long long, int>, "two pointers swapped");
static_assert(!takes<const int*, __nv_bfloat16*, long long, int>, "a pointer of another type");
static_assert(!takes<const float*, const __nv_bfloat16*, long long, int>, "const dropped");
static_assert(!takes<const float*, __nv_bfloat16*, float*, int>, "a pointer for a size");
static_assert(!takes<unsigned long, __nv_bfloat16*, long long, int>, "a number for a pointer");
"""


def test_a_chained_launch_checks_the_types_of_its_arguments(tmp_path):
    try:
        nvcc = build.nvcc_path()
    except RuntimeError:
        pytest.skip("no nvcc on this machine")
    source = tmp_path / "launches.cu"
    source.write_text(LAUNCHES)
    done = subprocess.run([nvcc, *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC, "-c",
                           str(source), "-o", str(tmp_path / "launches.o")], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert done.returncode == 0, done.stdout


def kernels():
    """``(name, body)`` of every kernel in the sources, and the names of those that are launched with <<<>>>."""
    found, ordinary = [], set()
    for name in build.SOURCES:
        with open(os.path.join(build.CSRC, name)) as file:
            text = re.sub(r"//[^\n]*", "", file.read())
        ordinary |= set(re.findall(r"(\w+)\s*(?:<[^;{}<>]*>)?\s*<<<", text))
        for match in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
            start = position = text.index("{", match.end())
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[position], 0)
                position += 1
                if depth == 0:
                    break
            found.append((match.group(1), text[start + 1:position - 1]))
        assert len(re.findall(r"__global__", text)) == len(re.findall(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?\w+\s*\(", text)), name
    return found, ordinary


def test_every_kernel_of_the_chain_waits_before_it_works_or_leaves():
    found, ordinary = kernels()
    chained = [(name, body) for name, body in found if name not in ordinary]
    assert len(chained) > 40 and ordinary
    late = []
    for name, body in chained:
        body = re.sub(r"\[&\]\([^)]*\)\s*\{[^{}]*\}", "", body)           # what a lambda returns leaves no kernel
        if "chain_begin();" in body:
            good = body.lstrip().startswith("chain_begin();")
        else:   # set up first: no way out and no status word written before the wait, and the next one let go only behind it
            wait = body.find("chain_wait();")
            good = wait >= 0 and not re.search(r"\breturn\b|atomicExch|chain_next", body[:wait])
        if not good:
            late.append(name)
    assert not late


def test_no_load_is_declared_free_of_order():
    """``__ldg`` promises that nobody writes the value while the kernel lives; in a chain its life begins before the writer's ends,
    and only the wait lies between them."""
    for name in sorted(os.listdir(build.CSRC)):
        with open(os.path.join(build.CSRC, name)) as file:
            text = re.sub(r"//[^\n]*", "", file.read())
        assert "__ldg" not in text, name
        assert re.findall(r'asm\s*\(\s*"ld\.', text) == [], name      # loads in inline PTX are volatile: they keep their place behind the wait


def test_what_is_read_ahead_of_a_wait_comes_from_the_l2():
    """A kernel that may read before it waits: what griddepcontrol.wait makes visible is promised to the grid that waited, and a line that
    an SM kept from an earlier kernel is none of it.  Such reads name the L2, where the writes of a completed kernel are."""
    found, _ = kernels()
    early = [(name, body[:body.rfind("chain_wait();")]) for name, body in found if re.search(r"if \([^;{}]*\)\s*chain_wait\(\);", body)]
    assert [name for name, _ in early] == ["stream_gemm_kernel"]
    for name, before in early:
        assert "load_l2(p.counts + " in before and "load_l2(p.offsets + " in before, name
        assert re.findall(r"\bp\.\w+\[", before) == [], name
