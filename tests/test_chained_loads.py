"""A chained kernel may be resident while its predecessor still writes what it reads, so every kernel that launch_chained()
starts waits first and reads through ordinary loads: no `const ... __restrict__` pointer and no read-only load intrinsic,
which are allowed to return the values of the kernel's start.  A race of this kind is not for a GPU to show: the sources
are read here."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deers_b200", "csrc")


def sources():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        out[os.path.basename(path)] = text
    return out


def kernels(text):
    """(name, parameter list, body up to the first statements) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1], text[i:i + 4000]


FILES = sources()
CHAINED = [(f, name, params, body) for f, text in FILES.items() if "launch_chained(" in text and f != "common.cuh"
           for name, params, body in kernels(text)]


def test_every_kernel_of_the_chained_files_is_seen():
    names = {name for _, name, _, _ in CHAINED}
    assert {"embedding_fwd_kernel", "rmsnorm_kernel", "rope_pack_kernel", "adamw_kernel", "attn_fwd_f16_kernel", "attn_bwd_f32_kernel",
            "attn_bwd_prep_f16_kernel", "attn_bwd_dkdv_f16_kernel", "gemm_f32_kernel", "gemm_f16x3_kernel", "gemm_f16_kernel",
            "decode_vec_kernel", "copy_logits_kernel", "x3_split_kernel"} <= names
    for text in FILES.values():
        for m in re.finditer(r"launch_chained\(ctx,\s*(\w+)", text):
            assert m.group(1) in names | {"kernel"}, m.group(1)


@pytest.mark.parametrize("file,name,params,body", CHAINED, ids=[f"{f}:{n}" for f, n, _, _ in CHAINED])
def test_chained_kernels_wait_and_read_coherently(file, name, params, body):
    assert not re.search(r"const\s+[\w ]+\*\s*__restrict__", params), f"{name}: read-only restrict parameter"
    head = body[:body.index(";", body.index("chain_"))] if "chain_" in body else ""
    assert re.search(r"chain_(next|wait|begin)\(\)", head), f"{name}: no wait"
    wait = re.search(r"chain_(wait|begin)\(\);", body)
    assert wait and not re.search(r"\*|\[", body[:wait.start()].split("{", 1)[1]), f"{name}: something precedes the wait"


@pytest.mark.parametrize("file", sorted(FILES))
def test_no_read_only_loads(file):
    assert not re.search(r"__ldg\(|__ldcs\(|__ldca\(|ld\.global(\.\w+)*\.nc", FILES[file]), file
    # locals of kernels: a restrict pointer to const data taken from a parameter structure
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+\w+\s*=", FILES[file]), file


@pytest.mark.parametrize("file", sorted(f for f in FILES if f.endswith(".cu")))
def test_refused_launches_end_the_call(file):
    """Behind a launch that was refused, the next kernel would work on what has not been written."""
    for m in re.finditer(r"launch_chained\(", FILES[file]):
        assert FILES[file][:m.start()].rstrip().endswith("DEERS_CUDA_TRY(ctx,"), FILES[file][m.start():m.start() + 80]


def test_rotation_promises_nothing_about_its_buffers():
    """The model rotates in place: source and destination are one buffer, which a restrict pointer to either would deny."""
    (body,) = [body for f, name, _, body in CHAINED if name == "rope_pack_kernel"]
    assert "p.dst" in body and "__restrict__" not in body
