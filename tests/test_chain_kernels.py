"""Kernels that can be launched early read what the chain hands on coherently.

A kernel launched by ``launch_early`` is resident while its predecessor still
writes.  The read-only path (``__ldg``, ``ldv``, const pointers with
``__restrict__``) asks for memory that nothing writes meanwhile, so it is open
only to arrays that are made before the chain starts.
"""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "redbirdpy_b200" / "csrc"
# made before the first early launch of a chain and not written by its kernels
CONSTANT = {"indptr", "indices", "val", "agg", "agg_ptr", "agg_rows", "is1", "rowscale", "par", "os", "cu", "cw", "cg",
            "B"}


def _kernels():
    """(name, parameters, body) of every kernel that waits for its predecessor."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        for m in re.finditer(r"__global__[^;{]*?(\w+)\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            body = text[m.end():i]
            if "chain_wait()" in body:
                yield m.group(1), m.group(2), body


def test_chain_kernels_read_handed_on_arrays_coherently():
    seen = []
    for name, params, body in _kernels():
        seen.append(name)
        for p in params.split(","):
            if "const" in p and "__restrict__" in p:
                assert p.split("__restrict__")[1].strip() in CONSTANT, (name, p.strip())
        # (spmm_kernel picks its load by type, in ldx)
        for call in re.findall(r"(?:\bldv<[^;]*|__ldg)\([^;]*;", re.sub(r"auto ldx = .*?\};\n", "", body, flags=re.S)):
            raise AssertionError((name, call))
    assert {"spmm_kernel", "spmm_pair_kernel", "gemm_tn_kernel", "gj_diag_kernel", "vc_spmm_kernel",
            "vc_pupdate_kernel", "vc_update_kernel", "vc_mid_spmm_kernel", "vc_prolong_kernel"} <= set(seen), seen


def test_chain_waits_come_first():
    for name, _, body in _kernels():
        before = re.sub(r"constexpr [^;]*;", "", body.split("chain_wait()")[0])
        assert not re.search(r"\[|\*\w|->", re.sub(r"__shared__[^;]*;", "", before)), (name, before)


def test_live_counts_are_read_through_l1():
    """Every warp of every iteration kernel reads the live count: a C++
    volatile read passes L1 by; an ordinary load in ordered assembly does not."""
    body = (CSRC / "rb_common.cuh").read_text().split("bool chain_dead(")[1].split("\n}")[0]
    assert "volatile int32_t" not in body and "asm volatile(\"ld.global.b32" in body
