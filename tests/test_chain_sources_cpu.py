"""Kernels of a dependent chain read what earlier kernels of the chain write through ordinary
loads only: read from the sources, because a violation is a race that no output has to show."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aethergraph_b200", "csrc")


def _balanced(text, start, pair):
    """End of the bracket that opens at `start`."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced source")


def _kernels(path):
    """(name, parameters, body) of every kernel in the file, comments removed."""
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*)?", text):
        at = m.end()
        if text[at] == "(":  # the launch bounds
            at = _balanced(text, at, "()")
        name = re.match(r"\s*(\w+)\s*", text[at:])
        params = at + name.end()
        end = _balanced(text, params, "()")
        body = text.index("{", end)
        yield name.group(1), text[params:end], text[body:_balanced(text, body, "{}")]


def _chained():
    for file in sorted(os.listdir(CSRC)):
        if file.endswith(".cu"):
            for name, params, body in _kernels(os.path.join(CSRC, file)):
                if "chain_sync()" in body:
                    yield pytest.param(params, body, id=f"{file}:{name}")


@pytest.mark.parametrize("params,body", list(_chained()))
def test_no_read_only_view_of_chain_data(params, body):
    assert "__restrict__" not in params and "__restrict__" not in body
    before = body[:body.index("chain_sync()")]
    assert not re.search(r"\bpa\b|\bgroup\b", before), "chain data is read before the wait"


def test_the_chains_kernels_are_found():
    assert len(list(_chained())) >= 10


@pytest.mark.parametrize("file,kernel,observed,read,order", [
    ("hetero.cu", "k_class_rank", "ld_acquire_u32(tiles", "__ldcg(d", r"__syncwarp\(\)"),
    ("sampler.cu", "k_pick_hub_slices", "atomicAdd(p.hub_done", "__ldcg(p.hub_key", r"__threadfence\(\).*__syncwarp\(\)"),
    ("rewrite.cu", "k_induce_walk", "atomicAdd((unsigned long long *)(a.total", "__ldcg(a.block_start", r"__threadfence\(\).*?__syncthreads\(\)"),
])
def test_what_one_thread_observes_is_passed_on_by_a_barrier(file, kernel, observed, read, order):
    """One thread sees that data is complete, others read it: its acquire (or fence) has to come
    before their reads through a barrier; a vote or a shuffle orders no memory."""
    body = next(b for n, _, b in _kernels(os.path.join(CSRC, file)) if n == kernel)
    at = body.index(observed)
    between = body[at:body.index(read, at)]
    assert re.search(order, between, re.S), between
