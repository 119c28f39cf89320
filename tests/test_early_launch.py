"""Kernels that may begin while the one before them still runs (programmatic launch) do not declare
what that one may write as read-only: the read-only path is specified for data that stays the same
while the kernel runs (no GPU; reads the sources)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tritonops_b200", "csrc")
READ_ONLY = re.compile(r"\bconst\s+\w+\s*\*\s*__restrict__|\bld_nc_16\b|\b__ldg\b|ld\.global\.nc")


def functions(src):
    """(name, text from the parameters to the closing brace) of every function of a source file."""
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)
    for m in re.finditer(r"\b(\w+)\s*(\((?:[^()]|\([^()]*\))*\))\s*\{", src):
        depth, i = 1, m.end()
        while depth and i < len(src):
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(1), src[m.start(2):i]


def test_nothing_is_read_as_constant_behind_an_early_launch():
    found, helpers = {}, {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        for name, text in functions(open(os.path.join(CSRC, f)).read()):
            if re.search(r"\bgrid_dependency_wait\(\);", text):
                found[name] = text
            else:
                helpers[name] = text
    for name in ("append_kernel", "bwd_rowsum_kernel", "bwd_convert_dq_kernel", "bwd_kernel", "prefill_kernel",
                 "decode_split_tma_kernel", "decode_combine_kernel", "rmsnorm_fwd_stream_kernel",
                 "rmsnorm_bwd_stream_kernel", "rmsnorm_dw_reduce_kernel"):
        assert name in found, name
    for name, text in found.items():
        assert not READ_ONLY.search(text), (name, READ_ONLY.search(text).group(0))
        for called in set(re.findall(r"\b(\w+)(?:<[\w, ]*>)?\(", text)) & set(helpers):   # one level: loads sit no deeper
            assert not READ_ONLY.search(helpers[called]), (name, called)
