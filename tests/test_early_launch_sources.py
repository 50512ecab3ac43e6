"""Kernels that may start before the launch in front of them has ended (pdl_wait) must not read their inputs through the
non-coherent path, nor have a load moved above the wait: checked in their source (csrc), on the CPU."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")


def functions(src):
    """(name, parameters, body) of every kernel and device function template at file level."""
    for m in re.finditer(r"^(\w+)\(((?:[^()]|\([^()]*\))*)\) \{\n(.*?)^\}\n", src, re.M | re.S):
        yield m.groups()


def test_early_launched_kernels_read_coherently_and_behind_the_wait():
    early = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            src = f.read()
        for name, params, body in functions(src):
            if "pdl_wait();" in body:
                early[name] = params
                assert not re.search(r"const \w+(?: \w+)?\* ?__restrict__", params), f"{name}: const __restrict__ input"
                assert not re.search(r"__ld(g|cs|cg|ca|lu)\(", body), f"{name}: load that the compiler may move"
    assert {"step_kernel", "gates_kernel", "gate_grad_anchored_kernel", "state_dot_kernel", "rec_body", "par_body"} <= set(early)
    with open(os.path.join(CSRC, "step.cu")) as f:
        vec4 = re.search(r"struct Vec4<float>.*?\n};\n.*?struct Vec4<__nv_bfloat16>.*?\n};\n", f.read(), re.S).group(0)
    assert "__ldcs" not in vec4
    with open(os.path.join(CSRC, "chunkwise_sm100.cu")) as f:
        assert "__restrict__" not in f.read()


def test_no_early_launched_kernel_is_overlooked():
    """Also those whose name stands behind __global__ on one line: every pdl_wait() is in a kernel that is looked at."""
    early, lets_in = {}, set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            src = f.read()
        waiting = [x for x in functions(src.replace(") par_", ")\npar_").replace(") part_kernel", ")\npart_kernel")) if "pdl_wait();" in x[2]]
        assert sum(body.count("pdl_wait();") for _, _, body in waiting) == src.count("pdl_wait();"), path
        for name, params, body in waiting:
            early[name] = params
            if "pdl_launch_dependents();" in body:
                lets_in.add(name)
            assert not re.search(r"const \w+(?: \w+)?\* ?__restrict__", params), f"{name}: const __restrict__ input"
            assert not re.search(r"__ld(g|cs|cg|ca|lu)\(", body), f"{name}: load that the compiler may move"
    assert {"step_kernel", "step_sequence_kernel", "gates_kernel", "gate_grad_rows_kernel", "gate_grad_scan_kernel",
            "gate_grad_anchored_kernel", "state_dot_kernel", "rec_body", "par_body", "par_bw_run_sm100", "part_kernel", "rec_scan_kernel",
            "par_fw_kernel", "par_bw_kernel"} <= set(early)
    # Kernels whose CTAs leave the next launch no room while they run, or that do the work of a call in a few of them, do not let
    # it in before they end: its CTAs would pile up where there is room at that moment.
    assert not {"par_bw_run_sm100", "part_kernel", "rec_scan_kernel", "par_fw_kernel", "par_bw_kernel"} & lets_in
    for name in ("chunkwise_bw_sm100.cu", "chunkwise_simt.cu"):   # (their device functions take the inputs in structs)
        with open(os.path.join(CSRC, name)) as f:
            assert "__restrict__" not in f.read(), name
