"""Kernels that may start under the tail of the kernel before them in the stream read what that kernel writes with ordinary
loads (ld_late), never by the read-only path, which is for data that no one writes while a kernel runs. A stale value would
show now and then at best, so the sources are held to it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "outbreaklab_b200", "csrc")

# kernel launched early: the functions that read for it, each with what the kernel before writes
LATE = {
    "ob_step.cu": {
        "k_advv2": {"advv2_body": ["F.Vt", "F.Vlo", "F.Vhi"], "sampleVt": ["F.Vt"]},
        "k_advq2": {"advq2_body": ["F.Qt"], "advq2_channel": ["F.Qt"], "box_channels": ["flagsB"]},
        "k_div": {"div_body": ["u", "v", "w"]},
        "k_proj": {"proj_body": ["F.phi"]},
    },
    "ob_dst_tc.cu": {
        "k_resid": {"resid_body": ["phi"], "k_resid": ["phi"]},
        "k_split_rows": {"k_split_rows": ["src", "p"]},
        # these read it by TMA, and the old values of an added sum through the pointer that they are stored by
        "k_dst_tc": {}, "k_dst_tc2": {}, "k_tri_tma": {},
    },
    "ob_mlp_train_tc.cu": {
        "k_mlp_step": {"k_mlp_step": ["bias", "P.w"]},
        "k_mlp_wgrad": {},   # by TMA
        "k_grad_adam": {"k_grad_adam": ["part"]},
    },
}


def _source(name):
    s = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", s)


def _function(src, name):
    """Signature and body of the function (the definition: its name, a parameter list, an opening brace)."""
    for m in re.finditer(r"\b%s\(" % name, src):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        j = i + len(src[i:]) - len(src[i:].lstrip())
        if src[j] != "{":
            continue
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        return src[m.start():k]
    raise AssertionError("no definition of " + name)


@pytest.mark.parametrize("name", sorted(LATE))
def test_every_early_kernel_is_listed(name):
    src = _source(name)
    calls = re.findall(r"launch_early\([^;]*;", src)
    early = {k for c in calls for k in re.findall(r"\bk_[a-z0-9_]+", c)}
    # k_split_rows' instances are picked into k first, k_dst_tc2 goes by pair_config
    early |= {"k_split_rows", "k_dst_tc2"} if name == "ob_dst_tc.cu" else set()
    assert early == set(LATE[name])


@pytest.mark.parametrize("name,kernel", [(f, k) for f in sorted(LATE) for k in LATE[f]])
def test_late_data_is_read_by_ordinary_loads(name, kernel):
    src = _source(name)
    assert "grid_wait()" in _function(src, kernel) or kernel in ("k_dst_tc", "k_tri_tma")   # those two wait in their bodies
    for fn, names in LATE[name][kernel].items():
        body = _function(src, fn)
        for n in names:
            e = re.escape(n)
            for load in ("__ldg", "ldo", "gather8", "gatherQ", "sampleVch", "trilerpB"):
                assert not re.search(r"\b%s\(\s*(reinterpret_cast<[^>]*>\(\s*)?%s\b" % (load, e), body), (fn, load, n)
            assert not re.search(r"__restrict__\s+%s\b" % e, body), (fn, n)
            if "." not in n and n not in ("src", "p"):
                assert not re.search(r"(?<![.\w])%s\[" % e, body), (fn, n)
