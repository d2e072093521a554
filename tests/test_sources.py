"""Rules of the kernels' sources that no result shows."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "visualmesh_b200", "csrc")

# what is in memory before the layer in front of a kernel begins: weights, neighbourhood, tile plan
CONSTANT = re.compile(r"(a\.(nb|weights|biases)|t\.bias|plan\.(halo_rows|halo_count)|h_rows|g|from|w|wp)\b")


def _kernels(text):
    """Bodies of the __global__ functions by name."""
    for begin in re.finditer(r"__global__ void [^;{]*?(\w+)\((?=const )", text):
        at = text.index("{", begin.end())
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield begin.group(1), text[at:end]


def _argument(text, at):
    depth, end = 1, at
    while depth:
        depth += {"(": 1, ")": -1}.get(text[end], 0)
        end += 1
    return text[at:end - 1]


def test_kernels_that_start_early_read_no_features_by_the_read_only_path():
    """Such a kernel runs while the layer in front of it still writes its input, and ld.global.nc is for what nobody writes meanwhile."""
    seen = set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cuh"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        for kernel, body in _kernels(text):
            if "after_previous(" not in body:
                continue
            seen.add(kernel)
            assert "ld.global.nc" not in body and "const __restrict__" not in body, kernel
            for load in re.finditer(r"__ldg\(", body):
                argument = re.sub(r"^reinterpret_cast<[^>]*>\(", "", _argument(body, load.end()))
                assert CONSTANT.match(argument), f"{kernel}: __ldg({argument})"
    assert seen == {"k_graph_conv_cw", "k_graph_conv_mma", "k_graph_conv_window"}


def test_a_layer_runs_on_the_kernel_whose_layout_its_input_has():
    """A kind of layer gets its features in a layout of its own, so no other kind's kernel, nor the CUDA cores', may take its place."""
    with open(os.path.join(CSRC, "engine.cu")) as f:
        text = f.read()
    begin = text.index("{", text.index("static void launch_conv("))
    body = _argument(text.replace("{", "(").replace("}", ")"), begin + 1)
    calls = list(re.finditer(r"launch_conv_(\w+)\(", body))
    assert {c.group(1) for c in calls} == {"window", "staged", "tc_split", "tc_gather", "ffma"}
    for call in calls:
        kind = {"window": "TC_WINDOW", "staged": "TC_STAGED"}.get(call.group(1), call.group(1).upper())
        line = body[body.rindex("case ", 0, call.start()):call.start()] if "case " in body[:call.start()] else body[:call.start()]
        assert re.findall(r"CONV_(\w+)", line) == [kind], call.group(0)
    assert "throw" in body[calls[-1].end():]
