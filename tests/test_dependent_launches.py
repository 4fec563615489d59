"""Kernels that may start before the previous kernel on the stream has ended
(programmatic dependent launches) read nothing that kernel may have written
ahead of their griddepcontrol.wait.  A reading of the sources: a kernel that
breaks the rule is wrong only now and then, and only on a device."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "self_b200", "csrc")
# inputs that no kernel of the call writes
INPUTS = {("k_grad", "feat"), ("k_grad", "label")}
# members of the argument structures that hold values, not addresses
VALUES = {"dgM", "bM", "bMf", "qw", "T", "nEl", "mode"}


def dependent_kernels():
    """(name, parameter list, body up to the wait, whole body) of every kernel that waits for its predecessor."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, f)).read(), flags=re.S)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?"
                             r"(\w+)\s*\(", src):
            def closing(at, left, right):
                depth = 0
                for k in range(at, len(src)):
                    depth += (src[k] == left) - (src[k] == right)
                    if depth == 0:
                        return k
            end = closing(m.end() - 1, "(", ")")
            opening = src.index("{", end)
            if src[end + 1:opening].strip():
                continue  # a declaration
            body = src[opening:closing(opening, "{", "}")]
            wait = re.search(r"griddepcontrol\.wait|after_previous\(\)", body)
            if wait:
                yield m.group(1), src[m.end():end], body[:wait.start()], body


def test_every_dependent_kernel_is_found():
    names = {k[0] for k in dependent_kernels()}
    assert {"k_grad", "k_adam", "k_entropy", "k_av_nu", "k_av_grad", "k_fused_stage_tma", "k_gradient",
            "k_vector_dg_divergence", "k_boundary_interp", "k_cig_llf"} <= names
    assert len(names) >= 40


def test_nothing_is_read_before_the_wait():
    for name, params, before, _ in dependent_kernels():
        for p in re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params):
            assert (name, p) in INPUTS or not re.search(rf"\b{p}\b", before), (name, p)
        for s in re.findall(r"(?:StageArgs|AvArgs)\s+(\w+)", params):
            assert set(re.findall(rf"\b{s}\.(\w+)", before)) <= VALUES, name


def test_no_pointer_of_a_dependent_kernel_is_restrict():
    """__restrict__ promises that nobody else writes the data while the kernel runs, but its run overlaps the kernel
    that writes it: the compiler could read it through the non-coherent path or move a read ahead of the wait."""
    for name, params, _, body in dependent_kernels():
        assert "__restrict__" not in params and "__restrict__" not in body, name
