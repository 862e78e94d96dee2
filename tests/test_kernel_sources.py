"""Rules that the CUDA sources keep and that no run would show reliably."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "lorax_b200" / "csrc" / "kernels"
# what kernels read without any kernel writing it: weights, biases, scales, adapters, embedding tables, tables of angles
CONSTANT_PARAMS = {"w", "b", "bias", "wr", "mu", "q", "sw", "table", "pos", "cos_sin"}
CONSTANT_LOADS = re.compile(r"__ldg\((reinterpret_cast<const (uint4|float4)\*>\()?(cs\b|a0 \+|a1 \+|wr \+|B \+|arow \+)")


def _sources():
    for path in sorted([*KERNELS.glob("*.cu"), *KERNELS.glob("*.cuh")]):
        yield path.name, re.sub(r"//[^\n]*", "", path.read_text())


def _kernels():
    for name, text in _sources():
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(([^{;]*?)\)\s*\{", text, re.S):
            depth, end = 1, m.end()
            while depth:
                depth += (text[end] == "{") - (text[end] == "}")
                end += 1
            yield f"{name}:{m.group(1)}", m.group(2), text[m.end():end]


def test_output_of_the_kernel_in_front_is_not_read_as_constant():
    """A kernel that is set up under its predecessor reads what kernels write with ordinary loads behind its wait: no `const __restrict__`
    parameter and no __ldg for anything but constants."""
    seen = 0
    for kernel, params, body in _kernels():
        if "pdl_wait" not in body:
            continue
        seen += 1
        read_only = {p.split()[-1] for p in params.split(",") if re.search(r"\bconst\b.*__restrict__", p)}
        assert read_only <= CONSTANT_PARAMS, (kernel, read_only - CONSTANT_PARAMS)
    assert seen > 40
    for name, text in _sources():
        for line in text.splitlines():
            assert line.count("__ldg(") == len(CONSTANT_LOADS.findall(line)), (name, line.strip())


def test_triggers_stand_behind_the_wait():
    for kernel, _, body in _kernels():
        at = [body.find(f) for f in ("pdl_trigger()", "pdl_launch_dependents()") if f in body]
        assert not at or 0 <= body.find("pdl_wait()") < min(at) or "shrink_rows_part" in body, kernel


def test_triggers_ahead_of_the_wait_are_asked_for():
    """Only launches that say so trigger in front of their wait: those of a model's step, whose first kernel waits before it triggers.  By default
    what a caller's kernels wrote two launches in front of a product is there when it reads its weights."""
    import inspect

    from lorax_b200.ops import native, reference
    ahead = {kernel.split(":")[1] for kernel, params, body in _kernels() if "pdl_wait_ahead(" in body}
    assert ahead == {"norm_residual_kernel", "rope_kvwrite_kernel", "act_mul_kernel", "attn_decode_kernel", "attn_combine_kernel"}
    for kernel, params, body in _kernels():
        calls = re.findall(r"pdl_wait_ahead\((.*?)\);", body)
        assert calls in ([], ["ahead"], ["p.ahead"]) and ("pdl_wait" in body or "pdl_trigger" not in body), kernel
        if "embed_kernel" in kernel or "embed_peer" in kernel or "embed_stream" in kernel:
            assert not calls, kernel
    for name in ("norm_residual", "rope_kvwrite", "act_mul", "attn_decode"):
        for ops in (native, reference):
            assert inspect.signature(getattr(ops, name)).parameters["ahead"].default is False, name


@pytest.mark.parametrize("T,N,K,parts", [
    (13, 4096, 4096, 4), (32, 4096, 2048, 4), (1, 4096, 1984, 1), (13, 6144, 4096, 3), (16, 5504, 1536, 3), (16, 5504, 1472, 1), (17, 5504, 3072, 3),
    (17, 5504, 3008, 1), (13, 8192, 2048, 2), (13, 9216, 1984, 1), (32, 8192, 3072, 2), (32, 8192, 3008, 1),
    (32, 4736, 4096, 1), (1, 9472, 4096, 1), (33, 4096, 4096, 1), (1, 4864, 4096, 1)])      # as many parts as SMs; 33 tokens; 114 of 148 SMs
def test_classic_split_only_where_it_measured_quicker(T, N, K, parts):
    from lorax_b200.ops import native
    assert native.gemm_plan(T, N, K)["split"] == parts


@pytest.mark.parametrize("r", [16, 64])
@pytest.mark.parametrize("N", [128, 256, 320, 384, 448, 896, 1600, 2880, 4096])
def test_prefetches_of_adapter_rows_stay_inside(N, r):
    """A pair of CTAs covers 256 features, 128 each: past the last feature there is nothing to fetch, and what the tiles fetch is B_cat once."""
    from lorax_b200.ops import native
    sizes = [native.load().lx_lora_tile_bytes(N, tile, r) for tile in range((N + 255) // 256 * 2)]
    assert sum(sizes) == N * r * 2
    assert all(size % 16 == 0 and tile * 128 * r * 2 + size <= N * r * 2 for tile, size in enumerate(sizes) if size)


@pytest.mark.parametrize("T,N,K,rank,taken", [
    (4001, 28672, 4096, 0, True), (256, 4096, 14336, 0, True), (512, 28672, 4096, 0, True),
    (1000, 4096, 256, 0, False), (2048, 512, 1024, 0, False), (320, 11008, 4096, 0, False), (193, 256, 64, 0, False),      # 20, 10, 29 % slower by pairs
    (256, 28672, 4096, 16, True), (4001, 4096, 4096, 32, True), (256, 6144, 4096, 16, True), (300, 4096, 14336, 32, True), (512, 1536, 4096, 16, False), (700, 6144, 4096, 16, False),
    (256, 11008, 4096, 0, True), (257, 6144, 4096, 0, False), (256, 6144, 1984, 0, False),
    (1000, 4096, 14336, 16, False), (800, 17920, 1536, 16, False), (200, 28672, 4096, 64, False)])                          # 10, 8, 6 %
def test_pairs_of_ctas_only_where_they_measured_quicker(T, N, K, rank, taken):
    import ctypes

    from lorax_b200.ops import native
    out = (ctypes.c_int * 4)()
    native.load().lx_gemm_pair_plan(T, N, K, 148, 74, 64 << 20, rank, out)
    assert (out[0] > 0) == taken
    native.load().lx_gemm_pair_plan(T, N, K, 148, 40, 64 << 20, rank, out)
    assert out[3] <= 40 and out[2] <= 40


@pytest.mark.parametrize("units,K,parts", [(1, 14336, 14), (24, 14336, 6), (72, 14336, 2), (74, 14336, 2), (75, 14336, 1), (3, 4096, 4), (36, 4096, 4), (48, 4096, 3), (72, 4096, 2), (75, 4096, 1),
                                           (1, 1536, 1), (12, 1536, 1), (1, 2880, 3), (50, 2880, 1), (2, 3080, 4), (0, 4096, 1)])      # 1536: two batches, 4096: four
def test_shrink_units_share_their_k_only_where_it_measured_quicker(units, K, parts):
    from lorax_b200.ops import native
    assert native.load().lx_lora_fused_k_parts(148, units, K) == parts


def test_pairs_of_ctas_stay_on_the_sms_they_are_given():
    """As many as run at the same time and no more than the launch's SMs hold, in both users; a plan is made for that number."""
    from lorax_b200.ops import native
    assert [native.load().lx_pairs_on(*a) for a in ((148, 74), (148, 70), (100, 74), (21, 74), (1, 74), (148, 0))] == [74, 70, 50, 10, 0, 0]
    for name in ("gemm_bf16.cu", "moe.cu"):
        text = (KERNELS / name).read_text()
        assert "pairs_on(num_sms, fit)" in text and "if (fit < 0) return fit;" in text


@pytest.mark.parametrize("avg_rows,n_w,K,act,pairs", [(192, 256, 64, "", 1), (191, 4096, 4096, "", 0), (700, 384, 4096, "", 0), (300, 512, 256, "relu2", 1), (300, 28672, 4096, "swiglu", 1),
                                                      (300, 4096, 3072, "swiglu", 1), (300, 2816, 2048, "swiglu", 0), (192, 512, 1024, "swiglu", 0)])      # 6 and 20 % slower by pairs
def test_expert_products_by_pairs_only_where_they_measured_quicker(avg_rows, n_w, K, act, pairs):
    from lorax_b200.ops import native
    assert native.load().lx_moe_by_pairs(avg_rows, n_w, K, native._MOE_ACTS[act]) == pairs


@pytest.mark.parametrize("form,T,N,entry,taken", [
    ("fp8", 32, 28672, 1, True), ("fp8", 64, 28672, 1, False), ("fp8", 256, 28672, 1, False), ("fp8", 96, 6144, 1, True), ("fp8", 160, 6144, 1, False), ("fp8", 144, 4096, 1, True),
    ("fp8", 256, 1536, 1, True), ("fp8", 257, 512, 1, False),
    ("fp8", 160, 6144, 7, False), ("fp8", 160, 6144, 8, True), ("fp8", 96, 28672, 32, True), ("fp8", 128, 28672, 32, False), ("fp8", 256, 6144, 16, True), ("fp8", 288, 6144, 32, False),
    ("wq4", 5, 28672, 1, True), ("wq4", 8, 28672, 1, True), ("wq4", 9, 28672, 1, False), ("wq4", 16, 6144, 1, True), ("wq4", 24, 6144, 1, False), ("wq4", 32, 4096, 1, True), ("wq4", 28, 28672, 14, True)])
def test_adapters_join_quantised_products_only_where_it_measured_quicker(monkeypatch, form, T, N, entry, taken):
    """Which steps ask the product's launch to add the adapters: read off what the wrappers ask for, with the library's calls left out."""
    import torch
    from types import SimpleNamespace as NS

    from lorax_b200.ops import native
    asked = []
    lib = NS(lx_lora_add_max_rows=native.load().lx_lora_add_max_rows, lx_gemm_fp8_block128=lambda *a: 0, lx_quant_act_fp8=lambda *a: 0, lx_wq4_gemm_lora=lambda *a: 0)
    ws = NS(gemm_ws=torch.empty(8), status=torch.empty(2), num_sms=148)
    for name, value in dict(load=lambda: lib, workspace=lambda dev: ws, _stream=lambda: None, _lora_expand=lambda out, lora: out,
                            _lora_add=lambda out, lora, quicker: asked.append(quicker)).items():
        monkeypatch.setattr(native, name, value)
    x, lora = torch.empty(T, 128, dtype=torch.bfloat16), (None, NS(num_tiles=-(-T // entry)))
    if form == "fp8":
        native.gemm_fp8(x, torch.empty(N, 128, dtype=torch.uint8), torch.empty(N // 128, 1), lora=lora)
    else:
        w = NS(shape=(N, 128), bits=4, table=None, group=128, perm=None, codes=torch.empty(1, dtype=torch.uint8), sz=torch.empty(1), int_zero=False)
        native.gemm_wq(x, w, lora=lora)
    assert asked == [taken]


@pytest.mark.parametrize("out,ldo,v,ldv", [(0x1004, 512, 0x2000, 192), (0x1000, 510, 0x2000, 192), (0x1000, 512, 0x2008, 192), (0x1000, 512, 0x2000, 190)])
def test_adapters_beside_quantised_products_are_refused_off_their_alignment(out, ldo, v, ldv):
    """Four results are written and four sums read at a time: what does not lie that way is refused before anything is launched."""
    import ctypes

    from lorax_b200.ops import native
    add = native.LxLoraAdd(0x3000, 1, 1, 0x4000, 0x5000, 0x6000, 0, v, ldv, 512, 512, 1, 0x7000)
    assert native.load().lx_gemm_fp8_block128(0x8000, 512, 0x9000, 16, 0xA000, 512, 0xB000, out, ldo, None, 1, 512, 512, None, 0, 0xC000, 148, 1, ctypes.byref(add), None) == -1001
    if v % 16 or ldv % 4:      # (the 4-bit kernel writes single results)
        assert native.load().lx_wq4_gemm_lora(0x8000, 512, 0x9000, 0xA000, None, out, ldo, 1, 512, 512, 128, 0, ctypes.byref(add), None) == -2
