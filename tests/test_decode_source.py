"""Rules of the decoding kernels that no run can show to be kept: a kernel launched while its predecessor still runs may not
declare the memory that the predecessor writes constant."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neuralnet.cpp_b200", "csrc", "decode.cu")
# written before a token's first kernel starts, or by no kernel: weights, norm parameters, biases, tables, the step's three integers
CONSTANT_DURING_A_TOKEN = {"W", "gamma", "beta", "bias", "rope", "step"}


def _kernels(src):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(((?:const|float|WT|int)[^{;]*)\)\s*\{", src):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        yield m.group(1), m.group(2), src[m.end():end]


def test_dependent_kernels_do_not_promise_constant_memory():
    src = open(SOURCE).read()
    dependent = [(name, params, body) for name, params, body in _kernels(src) if "pdl_wait()" in body]
    assert {name for name, _, _ in dependent} == {"gemv_kernel", "decode_attn_kernel"}
    for name, params, body in dependent:
        constant = {p.split()[-1] for p in params.split(",") if "const" in p.split() and "__restrict__" in p}
        assert constant <= CONSTANT_DURING_A_TOKEN, (name, constant - CONSTANT_DURING_A_TOKEN)
        # ... and reads none of it in front of the wait
        early = body[:body.index("pdl_wait()")]
        for produced in re.findall(r"const float\* (\w+)", params):
            assert not re.search(rf"(?<!<uintptr_t>\()\b{produced}\s*(\[|\+)", early), (name, produced)


def test_the_shortest_prompt_of_a_pass_is_the_same_for_host_and_library():
    import __graft_entry__ as entry
    assert int(re.search(r"constexpr int kPromptMin = (\d+);", open(SOURCE).read()).group(1)) == entry.load_package().trainer.PROMPT_MIN
