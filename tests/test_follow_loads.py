"""Kernels that start while the one before them ends (asv_follow) must not read that
one's output as read-only data, which the compiler may load ahead of the wait.
For every such kernel: the parameters that the launch before it can write, none of
them const __restrict__ or read by __ldg.  (Members of a struct of pointers are
plain loads.)"""
import os
import re

import pytest

# file -> kernel -> {parameter: names derived from it in the body}
CHAINS = {
    "asv_flow.cu": {
        "k_fl_gray": {}, "k_fl_down": {"in": ["src"]}, "k_fl_poly_h": {"img": []}, "k_fl_poly_v": {"h": []},
        "k_fl_up": {"coarse": ["F", "G"]}, "k_fl_iter": {"fin": ["fx_in", "fy_in"]}, "k_fl_store": {"flow": []},
    },
    "asv_connect.cu": {
        "k_cc_tile": {}, "k_cc_union": {"par": []}, "k_cc_runs": {}, "k_cc_link": {"par": []}, "k_cc_flatten": {"par": [], "cnt": []},
        "k_cc_prefix": {"chunk": [], "count": []}, "k_cc_compact": {"chunk": []}, "k_cc_kept_count": {"rsize": []},
        "k_cc_nodes": {"chunk": []}, "k_cc_jump": {"node": []}, "k_cc_output": {"node": []},
    },
    "asv_volume.cu": {
        "k_pass_prepare": {}, "k_jfa": {"in": []}, "k_jfa_first": {}, "k_jfa_second": {}, "k_post_stats": {}, "k_post_chunk_max": {},
        "k_post_prefix": {}, "k_post_apply": {},
    },
    "asv_metric.cu": {"k_metric_self": {}, "k_metric_ring": {}, "k_metric_combine": {}},
    "asv_noalloc.cu": {"k_na_count": {}, "k_na_scan": {}, "k_na_apply": {}},
}
CALL = re.compile(r"\basv_follow(?:_wait)?\(\);")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(k_\w+)\s*\(([^)]*)\)\s*\{")


def _kernels(src):
    src = re.sub(r"//[^\n]*", "", src)
    found = [(m.start(), m[1], " ".join(m[2].split()), m.end()) for m in KERNEL.finditer(src)]
    ends = [f[0] for f in found[1:]] + [len(src)]
    return {name: (params, src[body:end]) for (_, name, params, body), end in zip(found, ends)}, src


@pytest.mark.parametrize("name", sorted(CHAINS))
def test_no_read_only_loads_of_the_launch_before(name):
    from anisotropic_supervoxel_gb300 import _build
    kernels, src = _kernels(open(os.path.join(_build.CSRC, name)).read())
    assert {k for k, (_, body) in kernels.items() if CALL.search(body)} == set(CHAINS[name])
    for kernel, written in CHAINS[name].items():
        params, _ = kernels[kernel]
        for p, derived in written.items():
            decl = [d.strip() for d in params.split(",") if re.search(r"\b%s$" % p, d.strip())]
            assert len(decl) == 1, (kernel, p)
            assert not ("const" in decl[0] and "__restrict__" in decl[0]), (kernel, decl[0])
            for n in [p] + derived:
                text = kernels[kernel][1] if n != "in" else src        # (`in` goes on to device functions)
                assert not re.search(r"__ldg\(\s*%s\b" % n, text), (kernel, n)
    assert "const int32_t *__restrict__ in" not in src


def test_every_chain_is_listed():
    from anisotropic_supervoxel_gb300 import _build
    for f in sorted(os.listdir(_build.CSRC)):
        if f.endswith(".cu") and CALL.search(re.sub(r"//[^\n]*", "", open(os.path.join(_build.CSRC, f)).read())):
            assert f in CHAINS, f
