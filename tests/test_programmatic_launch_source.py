"""CPU check of the kernels' side of the programmatic launches."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "demystification_dfn_b200", "csrc")


def kernels():
    """(name, body) of every kernel."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for part in text.split("__global__")[1:]:
            name = re.search(r"(\w+_kernel)\s*\(", part).group(1)
            start = end = part.index("{")
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(part[end], 0)
                end += 1
                if depth == 0:
                    break
            yield name, part[start:end]


def test_a_kernel_that_triggers_waits_first():
    """Otherwise what runs before the wait of the kernel after next could read
    results that are not there yet."""
    seen = [name for name, body in kernels() if "pdl_trigger()" in body]
    assert len(seen) >= 8
    for name, body in kernels():
        if "pdl_trigger()" in body:
            assert "pdl_wait()" in body[:body.index("pdl_trigger()")], name


def test_a_kernel_launched_with_the_attribute_waits():
    names = {name: body for name, body in kernels()}
    with open(os.path.join(CSRC, "dfn_b200.cu")) as f:
        direct = set(re.findall(r"launch_pdl\(\s*(\w+_kernel)", f.read()))
    assert {"hm_permute_kernel", "tc_pack_v_kernel", "s64_pack_v_kernel", "tc_gemm_persistent_kernel",
            "mlp_grad_kernel", "mlp_reduce_adam_kernel"} <= direct
    # the others go through a function pointer or a choice of instantiations
    for name in direct | {"gemv_tma_kernel", "s64_gemm_kernel", "friction_kernel", "commit_kernel"}:
        assert "pdl_wait()" in names[name], name
