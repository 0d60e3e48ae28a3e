"""Source rule of the chained kernels (programmatic dependent launches): what the
kernel just before writes is read by ld_fresh, never through the read-only path.
Such a kernel starts while the one before still writes, and the read-only path is
defined only for data that does not change over a kernel's lifetime; a wrong read
shows in a run by chance only, so the rule is checked where it is written."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "ek-pnp_b200", "csrc")


def functions(name, file):
    """Texts, signature to closing brace, of the definitions of `name`."""
    s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    out = []
    for m in re.finditer(r"\b%s\(" % name, s):
        head = re.match(r"[^;{}]*\)\s*\{", s[m.start():])
        if not head:  # a call or a declaration
            continue
        end, depth = m.start() + head.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(s[end], 0)
            end += 1
        out.append(s[m.start():end])
    assert out, (name, file)
    return out


# function, file, what the kernel before wrote
FRESH = [
    ("efield_at", "ek_lbm_f64.cu", "psi"),
    ("efield_f32", "ek_lbm_f32.cuh", "psif|psim"),
    ("fwd_rows_any_len", "ek_poisson.cu", "rhs|r0|r1"),
    ("fwd_rows", "ek_poisson.cu", "rhs"),
    ("fwd_rows_f64_k", "ek_poisson.cu", "rhs|r0|r1"),
    ("fwd_rows_f64", "ek_poisson.cu", "rhs"),
    ("fwd_rows_f32_k", "ek_poisson.cu", "rhsf|q0|q1"),
    ("solve_cluster_f64", "ek_poisson.cu", "rhs"),
    ("tridiag_part_len", "ek_poisson.cu", "spec"),
    ("tridiag_part_gen", "ek_poisson.cu", "spec"),
    ("mse_grad", "ek_mlp.cu", "y"),
]


@pytest.mark.parametrize("name,file,written", FRESH, ids=[f[0] for f in FRESH])
def test_written_values_are_read_fresh(name, file, written):
    for text in functions(name, file):
        assert not re.search(r"__restrict__\s+(%s)\b" % written, text)
        assert not re.search(r"__ldg\([^;]*\b(%s)\b" % written, text)


def test_kernels_that_are_not_chained():
    """The gather of a training iteration and Adam read what the kernel before wrote
    through the read-only path: ordinary launches."""
    s = open(os.path.join(CSRC, "ek_mlp.cu")).read()
    for kernel in ("gather_batch", "adam_update", "bias_grads", "pad_inputs"):
        assert kernel + "<<<" in s and "launch_pdl(" + kernel not in s, kernel


def test_psi_fluctuation_rows_are_read_fresh():
    s = open(os.path.join(CSRC, "ek_lbm_f32.cuh")).read()
    body = s[s.index("template <typename V> struct PsiRow"):]
    body = body[:body.index("template <typename V> struct PerX")]
    assert "ld_fresh" in body and "ld_pop" not in body and "ld_pair" not in body and "__ldg" not in body
    assert all("PsiRow<V>" in t and "Row<V, float>" not in t for t in functions("efield_f32", "ek_lbm_f32.cuh"))


def test_fresh_loads_are_coherent_and_ordered():
    texts = functions("ld_fresh", "ek_internal.h")
    assert len(texts) == 4
    for t in texts:
        assert 'asm volatile("ld.global.' in t and ".nc" not in t
