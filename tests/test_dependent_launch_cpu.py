"""Kernels that may start beside the one before them: what a CTA allocates of tensor memory it has before its first thread lets the next
kernel begin (the other order can hang a GPU), and it reads no operand in a way a compiler may move ahead of its wait.  Both are read from
the sources."""
import dataclasses
import os
import re

import pytest

from fasteq_b200 import _build
from fasteq_b200.codegen import u1d as gen
from fasteq_b200.prebuild import cwtp_spec

GENERATED = [("128x0e+128x1o", 3, "f32"), ("64x0e+64x1o", 3, "f32"), ("33x0e+33x1o", 2, "f32"), ("64x0e+64x1o", 2, "f64")]


def _kernels():
    for name in _build.CORE_SOURCES:
        with open(os.path.join(_build.CSRC, name)) as f:
            yield name, f.read()
    for in1, lmax, dtype in GENERATED:
        spec = cwtp_spec(in1, lmax, lmax, dtype)
        for dual in ((), (True, True, True)):
            sp = dataclasses.replace(spec, dual=dual)
            yield f"{in1} {dual}", gen.emit_backward(sp, gen.untuned(sp, "bwd"), True, True, True)


@pytest.mark.parametrize("name,text", list(_kernels()), ids=[n for n, _ in _kernels()])
def test_tensor_memory_is_allocated_before_the_next_kernel_may_begin(name, text):
    for kernel in re.split(r"__global__", text)[1:]:
        alloc = re.search(r"tmem_alloc\(|tcgen05\.alloc", kernel)
        enter = re.search(r"wait_for_previous_kernel\(\)|let_next_kernel_begin\(\)", kernel)
        if alloc and enter:
            assert "__syncthreads()" in kernel[alloc.start():enter.start()]


@pytest.mark.parametrize("name", [n for n in _build.CORE_SOURCES])
def test_operands_are_read_after_the_wait(name):
    with open(os.path.join(_build.CSRC, name)) as f:
        text = f.read()
    for kernel in re.split(r"__global__", text)[1:]:
        body = kernel[:kernel.find("\n}\n")]
        if "wait_for_previous_kernel()" in body:
            assert "__ldg" not in body and "__restrict__" not in body[:body.find("{")]
