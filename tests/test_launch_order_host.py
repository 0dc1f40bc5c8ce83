"""What a kernel that begins while the one before it still runs (csrc/common.cuh: launch_early, follow_previous) may do, looked up in the
sources: loads marked read-only (`__ldg`, `ld.global.nc`) are defined only for memory that nobody writes during the kernel's whole life, and
the kernel before is still writing; and no thread leaves ahead of the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmq_b200", "csrc")


def functions(text):
    """(name, is a kernel, body) of every __global__ / __device__ function of a source without comments"""
    for m in re.finditer(r"__(global|device)__\b", text):
        at = text.find("{", m.end())
        head = text[m.end():at if at >= 0 else None]
        head = re.sub(r"__launch_bounds__\s*\([^()]*(?:\([^()]*\)[^()]*)*\)|__cluster_dims__\s*\([^()]*\)|__noinline__|__forceinline__", "", head)
        name = re.search(r"([A-Za-z_]\w*)\s*\(", head)
        if at < 0 or ";" in head or not name:
            continue
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield name.group(1), m.group(1) == "global", text[at:end]


def sources():
    found, calls = {}, []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                text = re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)
            calls.append(text)
            for name, kernel, body in functions(text):
                found.setdefault(name, []).append((f, kernel, body))
    return found, "\n".join(calls)


def early(found):
    return sorted({n for n, defs in found.items() for _, kernel, body in defs if kernel and "follow_previous(" in body})


def test_early_kernels_are_found():
    found, _ = sources()
    names = early(found)
    for n in ("gemm_skinny_kernel", "gemm_bf16_kernel", "gemm2_bf16_kernel", "gemm_grouped_kernel", "rmsnorm_kernel", "rope_kvwrite_kernel",
              "decode_attn_kernel", "prefill_attn_kernel", "prefill_tile_kernel", "argmax_kernel", "sample_kernel", "copy_f32_kernel",
              "moe_route_grouped_kernel", "residual_add_routed_v8_kernel", "silu_glu_v8_kernel", "swiglu_kernel", "gather_rows_kernel"):
        assert n in names, n


def test_no_read_only_loads_in_early_kernels():
    found, _ = sources()
    bad = []
    for kernel in early(found):
        seen, todo = set(), [kernel]
        while todo:
            name = todo.pop()
            if name in seen:
                continue
            seen.add(name)
            for f, _, body in found.get(name, ()):
                for word in ("__ldg", "ld_nc_v4", "ld.global.nc", "__ldcs", "ld.global.L1::no_allocate.nc"):
                    if re.search(re.escape(word) + r"\b", body) and name != "ld_nc_v4":
                        bad.append((kernel, f, name, word))
                todo += [c for c in re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^;{}()]*>)?\s*\(", body) if c in found]
    assert not bad, bad


def test_no_thread_leaves_ahead_of_the_wait():
    found, _ = sources()
    for kernel in early(found):
        for f, is_kernel, body in found[kernel]:
            if is_kernel and "follow_previous(" in body:
                wait = min(body.index(w) for w in ("follow_previous(", "wait_for_previous(") if w in body)
                # (a `return` of a lambda ahead of it does not end the kernel)
                ahead = re.sub(r"\[&?\]\s*\([^)]*\)\s*\{[^{}]*(?:\{[^{}]*\}[^{}]*)*\}", "", body[:wait])
                assert not re.search(r"\breturn\b", ahead), (f, kernel)
