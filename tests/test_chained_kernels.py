"""Kernels that may start while their predecessor in the stream still runs
(those that call grid_wait): none reads through a ``const __restrict__``
parameter, which states that the data stays as it is for the whole kernel,
except what no kernel of the stream writes near a chained launch: the model
parameters (copied in by zsme_set_params) and the preconditioner's factors
(formed two plain launches before).  Functions that they call with the
predecessor's data neither.  Source check, no GPU needed."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zoomy-dmplex_b200", "csrc")
STAYS = {"params", "lu", "piv", "rdiag"}
CALLED = {"face_contrib", "load_q", "imp_residual_cell", "finalize_cell", "finalize_deferred", "imp_finish_dots"}


def _functions():
    """(name, parameter list, body) of every function in the kernel headers."""
    for fn in sorted(os.listdir(CSRC)):
        if not fn.endswith(".cuh"):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, fn)).read()).replace("{}", "")
        for m in re.finditer(r"\b(\w+)\(([^(){};]*(?:\([^()]*\)[^(){};]*)*)\)\s*(?:const\s*)?\{", src):
            depth, i = 1, m.end()
            while depth and i < len(src):
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            yield m.group(1), m.group(2), src[m.end():i]


def _restricted_const(params):
    return {p for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)}


def test_chained_kernels_read_the_predecessor_through_plain_pointers():
    fns = list(_functions())
    chained = {n: p for n, p, body in fns if re.search(r"\bgrid_wait\(\)", body) and n.endswith("_kernel")}
    assert {"stage_kernel", "finalize_kernel", "step_tail_kernel", "imp_apply_kernel", "imp_multi_dot_kernel",
            "imp_project_kernel", "imp_normalize_kernel", "imp_perturb_kernel"} <= set(chained)
    called = [(n, p) for n, p, _ in fns if n in CALLED and "*" in p]
    assert {n for n, _ in called} >= CALLED - {"imp_finish_dots"}
    bad = {n: sorted(_restricted_const(p) - STAYS) for n, p in list(chained.items()) + called}
    assert not any(bad.values()), {n: b for n, b in bad.items() if b}
