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


def definitions(text):
    """{name: [(parameters, body)]} of the functions defined in a source."""
    out = {}
    for m in re.finditer(r"\b(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*(?:const\s*)?\{", text):
        if m.group(1) in ("if", "for", "while", "switch", "catch"):
            continue
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out.setdefault(m.group(1), []).append((m.group(2), text[m.end():i - 1]))
    return out


def reached(files, file, head):
    """Bodies of the functions a kernel calls before its wait, and of those they call: defined in its file, else in a header."""
    here = definitions(files[file])
    headers = {}
    for f, text in files.items():
        if f.endswith(".cuh"):
            for name, found in definitions(text).items():
                headers.setdefault(name, []).extend(found)
    seen, todo, out = set(), [head], []
    while todo:
        for name in re.findall(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\s*\(", todo.pop()):
            if name not in seen:
                seen.add(name)
                for params, body in here.get(name) or headers.get(name, []):
                    out.append((name, params, body))
                    todo.append(body)
    return out


def touches_global(files, file, head):
    """What a kernel's calls before the wait do that could reach global memory: an access through anything but shared memory and
    the arrays of a structure, or an instruction that loads, stores or copies outside shared memory."""
    arrays, found = set(), []
    text = files[file] + "".join(t for f, t in files.items() if f.endswith(".cuh") and f != file)
    for m in re.finditer(r"\bstruct\s+\w+\s*\{", text):                        # arrays that are members
        depth, members = 1, ""
        for c in text[m.end():]:
            depth += {"{": 1, "}": -1}.get(c, 0)
            if not depth:
                break
            members += c if depth == 1 else ""
        arrays |= set(re.findall(r"\b(\w+)\[[^\]]+\];", members))
    for name, params, body in reached(files, file, head):
        asm = " ".join(re.findall(r"asm\s*(?:volatile)?\s*\((.*?)\);", body, re.S))
        code = re.sub(r"asm\s*(?:volatile)?\s*\(.*?\);", "", body, flags=re.S)
        for ins in re.findall(r"(?:^|[\"\s;{])((?:ld|st|atom|red|cp|multimem|tcgen05\.(?:ld|st|cp|mma))\.[\w.:]+)", asm):
            if "global" in ins or ".shared" not in ins:
                found.append((name, ins))
        shared = set(re.findall(r"__shared__[^;]*?\b(\w+)\s*\[", code)) | set(re.findall(r"\b(?!return\b)\w+ (\w+)\[[^\]]+\];", code))
        for _ in range(3):                                       # pointers into it, and pointers from those
            for var, init in re.findall(r"\*\s*(?:const\s+)?(\w+)\s*=\s*([^;]*);", code):
                if set(re.findall(r"\w+", init)) & shared:
                    shared.add(var)
        for var in re.findall(r"(\w+)\s*\[", re.sub(r"__shared__[^;]*;", "", code)):
            if var not in shared | arrays and not re.search(r"\w+&?\s*\(&" + var + r"\)\[", params):
                found.append((name, var + "[]"))
        if re.search(r"\)\s*\[", code) or re.search(r"(?:^|[=(,;{}&|+\-!?:<>]|return)\s*\*\s*[\w(]", code) or "->" in code:
            found.append((name, "*"))
        found += [(name, f) for f in re.findall(r"\b(atomic\w+|__ld\w+|__st\w+)\s*\(", code)]
    return found


def head_of(body):
    """A kernel's text up to its wait."""
    return body[:re.search(r"chain_(wait|begin)\(\);", body).start()].split("{", 1)[1]


@pytest.mark.parametrize("file,name,params,body", CHAINED, ids=[f"{f}:{n}" for f, n, _, _ in CHAINED])
def test_what_runs_before_the_wait_stays_off_global_memory(file, name, params, body):
    assert touches_global(FILES, file, head_of(body)) == []


def test_calls_before_the_wait_are_followed():
    names = {n for f, _, _, body in CHAINED for n, _, _ in reached(FILES, f, head_of(body))}
    assert {"setup", "init", "row_of", "pick", "tile_m", "tile_n", "args", "attn_fwd_f16_prologue", "attn_bwd_dkdv_f16_prologue",
            "attn_bwd_dq_from_ds_f16_prologue", "gemm_f16_prologue", "gemm_f16x3_prologue", "mbar_init", "tmem_alloc",
            "tma_prefetch_desc"} <= names


@pytest.mark.parametrize("file,kernel,before,planted", [
    ("gemm_f32_kernel.cuh", "gemm_f32_kernel", "        base = b;\n", "        step = (long long)b[r0];\n"),
    ("gemm_f32_kernel.cuh", "gemm_f32_kernel", "        base = b;\n", "        step = *(b + r0);\n"),
    ("gemm_f32_kernel.cuh", "gemm_f32_kernel", "        base = b;\n", "        cp4(nullptr, b, 4);\n"),
    ("gemm_f32_kernel.cuh", "gemm_f32_kernel", "        base = b;\n", "        return b[r0];\n"),
    ("gemm_f32_kernel.cuh", "gemm_f32_kernel", "        kbeg = part * g.k_chunk;\n", "        if (g.a[0] > 0.f) return;\n"),
    ("gemm_f32.cu", "gemm_f32_group_kernel", "        int i = 0;\n", "        if (*g->c > 0.f) ++i;\n"),
    ("gemm_f16_sm100.cu", "gemm_f16_kernel", "        fence_barrier_init();\n", "        atomicCAS(err, 0u, 1u);\n"),
    ("gemm_f16_sm100.cu", "gemm_f16_kernel", "        fence_barrier_init();\n", "        tmem_base_s[2] = *(volatile unsigned int*)tmap_a;\n"),
    ("attn_fwd_f16_sm100.cu", "attn_fwd_f16_kernel", "        fence_barrier_init();\n", "        tmem_base_s[2] = ((const uint32_t*)tmap_q)[0];\n")])
def test_an_early_access_is_seen(file, kernel, before, planted):
    """The same sources with an access put into what runs before the wait (as text: nothing of it is built)."""
    assert before in FILES[file]
    files = dict(FILES, **{file: FILES[file].replace(before, before + planted)})
    heads = [head_of(body) for name, _, body in kernels(files[file]) if name == kernel]
    assert heads and all(touches_global(files, file, h) for h in heads)


@pytest.mark.parametrize("file", sorted(FILES))
def test_no_read_only_loads(file):
    assert not re.search(r"__ldg\(|__ldcs\(|__ldca\(|ld\.global(\.\w+)*\.nc", FILES[file]), file
    # locals of kernels: a restrict pointer to const data taken from a parameter structure
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+\w+\s*=", FILES[file]), file


@pytest.mark.parametrize("file", sorted(f for f in FILES if f != "common.cuh"))
def test_refused_launches_end_the_call(file):
    """Behind a launch that was refused, the next kernel would work on what has not been written."""
    for m in re.finditer(r"launch_chained\(", FILES[file]):
        assert FILES[file][:m.start()].rstrip().endswith("DEERS_CUDA_TRY(ctx,"), FILES[file][m.start():m.start() + 80]


@pytest.mark.parametrize("kernel", ["rope_pack_kernel", "cross_entropy_bwd_kernel"])
def test_kernels_that_work_in_place_promise_nothing_of_their_buffers(kernel):
    """Source and destination may be one buffer, which a restrict pointer to either would deny."""
    (found,) = [params + body[:body.index("__global__") if "__global__" in body else None] for f, name, params, body in CHAINED if name == kernel]
    assert re.search("p.dst|dlogits", found) and "__restrict__" not in found


def body_of(text, name):
    """The whole body of a kernel."""
    m = re.search(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?" + name + r"\s*\(", text)
    i = text.index("{", m.end())
    start, depth = i + 1, 1
    while depth:
        i += 1
        depth += {"{": 1, "}": -1}.get(text[i], 0)
    return text[start:i]


def closing(text, i):
    """Place of the bracket that closes the one at i."""
    depth, pair = 0, {"(": ")", "[": "]"}[text[i]]
    while True:
        depth += {text[i]: 0, "(": 1, "[": 1, ")": -1, "]": -1}.get(text[i], 0)
        if text[i] == pair and depth == 0:
            return i
        i += 1


def read_through(files, file, body, names):
    """Those of the pointers `names`, and of the pointers made from them, that a body dereferences other than as the target of an assignment, or
    hands to a function of the file that does."""
    out, todo, seen = [], list(names), set()
    while todo:
        p = todo.pop()
        if p in seen:
            continue
        seen.add(p)
        todo += re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*=[^;=]*\b" + p + r"\b", body)
        for m in re.finditer(r"\b" + p + r"\b", body):
            end, star = m.end(), re.search(r"(?:[;{}=(,]|\breturn)\s*\*\s*$", body[:m.start()])
            outer = [c for c in re.finditer(r"(\w+)(<[\w ]+\*>)?\(", body[:m.start()]) if closing(body, c.end() - 1) > m.start()]
            if not star and outer and outer[-1].group(1) == "reinterpret_cast":
                end = closing(body, outer[-1].end() - 1) + 1
                star = re.search(r"(?:[;{}=(,]|\breturn)\s*\*\s*$", body[:outer[-1].start()])
            elif outer:
                place = body[outer[-1].end():m.start()].count(",")
                for params, inner in definitions(files[file]).get(outer[-1].group(1), []):
                    if read_through(files, file, inner, [re.findall(r"(\w+)\s*(?:,|$)", params)[place]]):
                        out.append(p)
            after = body[end:].lstrip()
            if after.startswith("["):
                after = after[closing(after, 0) + 1:].lstrip()
            elif not star:
                continue
            if not re.match(r"=[^=]", after):
                out.append(p)
    return out


@pytest.mark.parametrize("file,name,params", [c[:3] for c in CHAINED if "__restrict__" in c[2]], ids=[f"{f}:{n}" for f, n, p, _ in CHAINED if "__restrict__" in p])
def test_restrict_pointers_of_chained_kernels_are_only_written(file, name, params):
    """The promise that nothing else reaches what a pointer points to lets a load through it run ahead of the wait, const or not."""
    names = re.findall(r"\*\s*__restrict__\s+(\w+)", params)
    assert read_through(FILES, file, body_of(FILES[file], name), names) == []


@pytest.mark.parametrize("file,kernel,before,planted", [
    ("rmsnorm.cu", "rmsnorm_kernel", "            acc = warp_sum(acc);\n", "            inv = inv_out[row];\n"),
    ("rmsnorm.cu", "rmsnorm_block_kernel", "        acc = warp_sum(acc);\n", "        acc += reinterpret_cast<const float4*>(out + row * C)[0].x;\n"),
    ("rmsnorm.cu", "rmsnorm_kernel", "    const float x[4] = {v.x, v.y, v.z, v.w};\n", "    const float y = __half2float(hi[at]);\n"),
    ("gpt_ops.cu", "cross_entropy_merge_kernel", "    lse[row] = l;\n", "    picked[row] = lse[row];\n"),
    ("gemm_f16x3_sm100.cu", "x3_split_kernel", "        __half* dh = hi + r * ld_dst + c0;\n", "        if (dh[0] == h[0]) continue;\n")])
def test_a_read_through_a_restrict_pointer_is_seen(file, kernel, before, planted):
    assert before in FILES[file]
    files = dict(FILES, **{file: FILES[file].replace(before, before + planted)})
    (params,) = [params for f, name, params, _ in CHAINED if name == kernel]
    assert read_through(files, file, body_of(files[file], kernel), re.findall(r"\*\s*__restrict__\s+(\w+)", params))


def test_no_restrict_locals_that_are_only_read():
    for file, text in FILES.items():
        for m in re.finditer(r"\*\s*__restrict__\s+(\w+)\s*=", text):
            rest = text[m.end():m.end() + 4000]
            assert re.search(r"(?:\*reinterpret_cast<\w+\*>\(" + m.group(1) + r"\b[^;]*\)|\b" + m.group(1) + r"\[[^\]]*\])\s*=[^=]", rest), (file, m.group(1))
