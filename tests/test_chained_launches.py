"""Kernels launched by launch_chained are placed while the launch before them still runs and wait for it
(griddepcontrol.wait).  The wait is an asm statement that read-only loads (__ldg, const __restrict__ arguments)
may be moved above, unless the address comes out of it: every array that a launch before writes and the kernel
loads that way has to pass through chain_wait or after_wait.  Read from the sources (a missing one shows no
error on most runs)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "city-scale-nlos-acoustic-engine-code_b200", "csrc")

# what the kernel loads through the read-only path and a launch directly before it may write
READS = {
    "k_step": {"fin"},                                    # the population buffer (any step, ghost fill, source)
    "k_step_a": {"fin"},
    "k_side_a": {"fin"},
    "k_source": {"f"},
    "k_ghost": {"f"},
    "k_adj_between": {"lam_in", "gadj", "face_mom"},      # adjoint step; itself; ghost fill of a recompute
    "k_adj_step": {"lam_in", "gadj"},                     # k_adj_between (residuals, ghost adjoints)
}


def kernels():
    """{name: (file text, body)} of the __global__ functions."""
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            at = text.index("{", m.end())
            depth, end = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out[m.group(1)] = (text, text[at:end])
    return out


def test_every_chained_kernel_waits_for_what_it_reads():
    ks = kernels()
    chained = {n for n, (text, _) in ks.items() for c in re.findall(r"launch_chained\((\w+)", text)
               if c == n or (c == "kernel" and re.search(r"kernel\s*=[^;]*\b%s\b" % n, text))}
    # (k_step_hw shares the name `kernel` with a chained one and is launched directly)
    assert chained - {"k_step_hw"} == set(READS)
    for name, arrays in READS.items():
        body = ks[name][1]
        waited = set(re.findall(r"\b(?:chain_wait|after_wait)\(\s*(?:\w+\.)*(\w+)\s*\)", body))
        assert arrays <= waited, (name, arrays - waited)


def test_a_refused_chained_launch_leaves_no_error_behind():
    """cudaLaunchKernelEx returns its error and keeps it as the last one too, where the next plain launch of any
    handle, which asks for the last error, would find it."""
    text = open(os.path.join(CSRC, "device.hpp")).read()
    body = text[text.index("cudaError_t launch_chained("):]
    body = body[:body.index("\n}\n")]
    assert "cudaLaunchKernelEx" in body and "cudaGetLastError()" in body
