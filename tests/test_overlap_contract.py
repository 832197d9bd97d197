"""Kernels that may start before the kernel ahead of them has ended (they call pdl_wait) must not take anything as
`const T* __restrict__`: that promises data read-only for the kernel's whole life, and lets the compiler load it before
the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sandbox_reactions_b200", "csrc")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(")


def kernels(text):
    heads = list(KERNEL.finditer(text))
    for k, m in enumerate(heads):
        end = heads[k + 1].start() if k + 1 < len(heads) else len(text)
        body = text.index("{", m.end())
        yield m.group(1), text[m.end():body], text[body:end].split("\n}\n")[0]


def test_overlapped_kernels_promise_nothing_of_their_inputs():
    overlapped = {}
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            for kernel, args, body in kernels(f.read()):
                if "pdl_wait()" in body:
                    overlapped[kernel] = args
    assert {"spmv_dir_kernel", "pcg_update4_kernel", "mg_tail_kernel", "mg_rowband_tma_kernel", "conv_tc_kernel",
            "hydro_band_kernel", "grav_columns_kernel", "grav_rows_inverse_kernel"} <= set(overlapped)
    for kernel, args in overlapped.items():
        assert not re.search(r"const[^,]*\*\s*__restrict__", args), kernel
