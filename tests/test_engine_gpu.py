"""GPU end-to-end: the bf16 kernel path must agree with the fp32 CPU oracle of the same model."""
import pytest
import torch

from lorax_b200.adapters.lora import random_adapter
from lorax_b200.adapters.manager import AdapterManager
from lorax_b200.config import EngineConfig, tiny_llama
from lorax_b200.models.decoder import DecoderModel
from lorax_b200.runtime.engine import Engine
from lorax_b200.runtime.kv_cache import KVCache
from lorax_b200.runtime.runner import ModelRunner, PrefillItem

pytestmark = pytest.mark.gpu

TARGETS = ["q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj"]


def _build(device, dtype, n_adapters=3):
    cfg = tiny_llama()
    model = DecoderModel.random_init(cfg, device, dtype, seed=0)
    mgr = AdapterManager(model, arena_bytes=64 << 20, host_bytes=128 << 20)
    for i in range(n_adapters):
        c, mm = random_adapter(cfg, r=[8, 16, 32][i % 3], alpha=16, target_modules=TARGETS, seed=10 + i, std_a=0.05, std_b=0.05)
        mgr.register(f"a{i}", c, mm)
        assert mgr.load(i + 1, f"a{i}")
    return cfg, model, mgr


def test_prefill_logits_match_cpu_oracle():
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    _, cm, _ = _build("cpu", torch.float32)
    g = torch.Generator().manual_seed(3)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (17, 64, 90)]
    outs = []
    for m in (gm, cm):
        kv = KVCache(cfg.num_hidden_layers, 32, m.nkv, m.d, m.dtype, m.device)
        r = ModelRunner(m, kv, max_batch=4, max_seq_tokens=256, max_prefill_tokens=512, use_graphs=False)
        items = [PrefillItem(p, 0, [1 + 3 * i, 2 + 3 * i, 3 + 3 * i], adapter_index=i) for i, p in enumerate(prompts)]
        _, _, logits = r.prefill(items)
        outs.append(logits.float().cpu())
    from lorax_b200.ops import native
    native.workspace().check_status()
    err = (outs[0] - outs[1]).norm() / outs[1].norm()
    assert err < 3e-2, err
    # the adapters change the logits by much more than the bf16 error
    assert (outs[1][1] - outs[1][0]).norm() > 0


def test_native_layers_take_adapters_that_come_after_the_first_step():
    """Prompts before any adapter is resident, with adapters, after the last one has left and with one again: the native layers give what
    the per-kernel path gives."""
    cfg, gm, mgr = _build("cuda", torch.bfloat16, 0)
    for i, r in enumerate([16, 32]):
        c, mm = random_adapter(cfg, r=r, alpha=16, target_modules=TARGETS, seed=40 + i, std_a=0.05, std_b=0.05)
        mgr.register(f"a{i}", c, mm)
    g = torch.Generator().manual_seed(12)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (17, 64, 33)]
    kv = KVCache(cfg.num_hidden_layers, 16, gm.nkv, gm.d, gm.dtype, gm.device)
    r = ModelRunner(gm, kv, max_batch=4, max_seq_tokens=128, max_prefill_tokens=256, use_graphs=False)
    blocks = [[1 + 3 * i + j for j in range(3)] for i in range(3)]

    def both(ads):
        out = []
        for gm.use_native_layers in (True, False):
            out.append(r.prefill([PrefillItem(p, 0, b, adapter_index=a) for p, b, a in zip(prompts, blocks, ads)])[2].clone())
        torch.cuda.synchronize()
        assert torch.equal(*out), ads
        return out[0]

    plain = both([0, 0, 0])
    executor = gm._native
    assert executor is not None and mgr.load(1, "a0") and mgr.load(2, "a1")
    with_adapters = both([1, 0, 2])
    assert torch.equal(with_adapters[1], plain[1])
    assert all((with_adapters[i] - plain[i]).norm() > 0.01 * plain[i].norm() for i in (0, 2))
    mgr.offload(1)
    mgr.offload(2)
    assert mgr.max_rank == 0 and torch.equal(both([0, 0, 0]), plain)
    assert mgr.load(2, "a1")
    again = both([2, 0, 0])
    assert gm._native is executor and (again[0] - plain[0]).norm() > 0.01 * plain[0].norm()


def test_native_layer_executor_equals_python_path():
    """The C++ layer executor issues the same kernels with the same arguments as the per-kernel Python path: prefill
    logits and a mixed prefill + decode step must be bit-identical."""
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    g = torch.Generator().manual_seed(11)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (17, 64, 90, 33)]
    results = []
    for native_on in (True, False):
        gm.use_native_layers = native_on
        kv = KVCache(cfg.num_hidden_layers, 64, gm.nkv, gm.d, gm.dtype, gm.device)
        r = ModelRunner(gm, kv, max_batch=8, max_seq_tokens=256, max_prefill_tokens=512, use_graphs=False)
        blocks = [[1 + 4 * i + j for j in range(4)] for i in range(4)]
        items = [PrefillItem(p, 0, blocks[i], adapter_index=i) for i, p in enumerate(prompts[:2])]
        ids, lps, logits = r.prefill(items)
        rows = [r.state.take_row(i) for i in range(2)]
        r.install(rows, ids, [len(p) for p in prompts[:2]], blocks[:2], [0, 1])
        r.resort()
        # prompts 2 and 3 ride along with the two decode rows
        k, nd, first_ids, first_lps = r.mixed_step([PrefillItem(p, 0, blocks[2 + i], adapter_index=2 + i) for i, p in enumerate(prompts[2:])])
        dec_ids, dec_lps = r.wait(k)
        torch.cuda.synchronize()
        results.append((logits.clone(), dec_ids[:nd].clone(), dec_lps[:nd].clone(), first_ids.clone(), first_lps.clone()))
        assert (gm._native is not None) == native_on or not native_on
    from lorax_b200.ops import native
    native.workspace().check_status()
    for a, b in zip(*results):
        assert torch.equal(a, b)
    gm.use_native_layers = True


def test_fp8_model_prefill_matches_cpu_oracle():
    """`quantize_fp8()` on both devices: the tcgen05 fp8 GEMM path against the PyTorch oracle of the same quantised
    model (same e4m3 weights and scales, activations rounded the same way), adapters included."""
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    _, cm, _ = _build("cpu", torch.float32)
    _, base, _ = _build("cpu", torch.float32)
    gm.quantize_fp8()
    cm.quantize_fp8()
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (9, 40, 70)]
    outs = []
    for m in (gm, cm, base):
        kv = KVCache(cfg.num_hidden_layers, 32, m.nkv, m.d, m.dtype, m.device)
        r = ModelRunner(m, kv, max_batch=4, max_seq_tokens=256, max_prefill_tokens=512, use_graphs=False)
        items = [PrefillItem(p, 0, [1 + 3 * i, 2 + 3 * i, 3 + 3 * i], adapter_index=i) for i, p in enumerate(prompts)]
        _, _, logits = r.prefill(items)
        outs.append(logits.float().cpu())
    from lorax_b200.ops import native
    native.workspace().check_status()
    # the two devices round activations that differ by bf16 noise, so some e4m3 roundings flip (one step = 6 %); what must
    # hold is that the GPU path is as close to the unquantised model as the oracle of the quantised model is
    e_gpu = ((outs[0] - outs[2]).norm() / outs[2].norm()).item()
    e_cpu = ((outs[1] - outs[2]).norm() / outs[2].norm()).item()
    assert e_cpu < 0.15 and e_gpu < 1.25 * e_cpu + 0.01, (e_gpu, e_cpu)
    assert (outs[0] - outs[1]).norm() / outs[1].norm() < 0.1


@pytest.mark.parametrize("graphs", [False, True])
def test_decode_logits_match_cpu_oracle_teacher_forced(graphs):
    """Prefill 8 requests over 4 adapters, then 12 decode steps; both devices are fed the oracle's tokens so
    that a near-tie flipped by bf16 cannot make the sequences diverge, and the logits are compared per step."""
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    _, cm, _ = _build("cpu", torch.float32)
    g = torch.Generator().manual_seed(4)
    prompts = [torch.randint(0, cfg.vocab_size, (int(torch.randint(16, 65, (1,), generator=g)),), generator=g).tolist() for _ in range(8)]
    ads = [i % 4 for i in range(8)]
    runners = []
    for m in (cm, gm):
        kv = KVCache(cfg.num_hidden_layers, 64, m.nkv, m.d, m.dtype, m.device)
        runners.append(ModelRunner(m, kv, max_batch=8, max_seq_tokens=256, max_prefill_tokens=1024, use_graphs=graphs))
    blocks = [[1 + 4 * i + j for j in range(4)] for i in range(8)]
    firsts = None
    for r in runners:
        items = [PrefillItem(p, 0, blocks[i], adapter_index=ads[i]) for i, p in enumerate(prompts)]
        ids, _, logits = r.prefill(items)
        if firsts is None:
            firsts = ids.tolist()
        rows = [r.state.take_row(i) for i in range(8)]
        r.install(rows, firsts, [len(p) for p in prompts], blocks, ads)
    worst = 0.0
    for step in range(12):
        outs = []
        for r in runners:
            k, b, logits = r.decode(need_logits=True)
            outs.append(logits[:8].float().cpu().clone())
        oracle_next = outs[0].argmax(-1).to(torch.int32)
        for r in runners:
            r.state.input_ids[:8].copy_(oracle_next.to(r.device))      # teacher forcing
        err = ((outs[1] - outs[0]).norm() / outs[0].norm()).item()
        worst = max(worst, err)
    from lorax_b200.ops import native
    native.workspace().check_status()
    assert worst < 3e-2, worst


@pytest.mark.parametrize("weights", ["bf16", "fp8", "gptq"])
def test_captured_steps_follow_the_largest_rank(weights):
    """Adapters of larger ranks that come after a batch's graph was captured, and smaller ones that are left: the step's launches cover the
    ranks that are there.  The same launches outside a graph give the same bits."""
    cfg, gm, _ = _build("cuda", torch.bfloat16, 0)
    if weights != "bf16":
        gm.quantize(weights)
    mgr = gm.adapters
    for i, r in enumerate([16, 32, 64]):
        c, mm = random_adapter(cfg, r=r, alpha=16, target_modules=TARGETS, seed=30 + i, std_a=0.05, std_b=0.05)
        mgr.register(f"a{i}", c, mm)
    g = torch.Generator().manual_seed(8)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (17, 40, 33)]
    blocks = [[1 + 2 * i, 2 + 2 * i] for i in range(3)]
    runners = [ModelRunner(gm, KVCache(cfg.num_hidden_layers, 8, gm.nkv, gm.d, gm.dtype, gm.device), max_batch=4, max_seq_tokens=64,
                           max_prefill_tokens=128, use_graphs=graphs) for graphs in (True, False)]

    def step(r, ads):
        for row in list(r.state.live):
            r.retire([row])
            r.state.drop_row(row)
        ids, _, _ = r.prefill([PrefillItem(p, 0, b, adapter_index=a) for p, b, a in zip(prompts, blocks, ads)])
        r.install([r.state.take_row(i) for i in range(3)], ids, [len(p) for p in prompts], blocks, ads)
        r.resort()
        logits = r.decode(need_logits=True)[2][:3].clone()
        torch.cuda.synchronize()
        return logits

    from lorax_b200.ops import native
    seen = []
    for ads in ([1, 0, 1], [2, 1, 2], [3, 2, 1], [1, 0, 1]):
        for a in ads:
            assert a == 0 or mgr.load(a, f"a{a - 1}")
        if len(seen) == 3:
            mgr.offload(3)
            mgr.offload(2)
        native.workspace().lora_v.fill_(3.0)                 # what a launch does not cover shows
        native.workspace().lora_vimg.fill_(3.0)
        got, want = (step(r, ads) for r in runners)
        assert torch.equal(got, want), ads
        seen.append(got)
    native.workspace().check_status()
    assert torch.equal(seen[0], seen[3]) and (seen[1] - seen[0]).norm() > 0.05 * seen[0].norm()


def test_adapter_copies_stay_out_of_captures():
    """However many managers a process makes, none copies on the stream that graphs are captured on: a pinned block of its copies may be
    released while a graph is captured, and pinned memory of its size is to be had afterwards."""
    cfg, gm, mgr = _build("cuda", torch.bfloat16, 1)
    r = ModelRunner(gm, KVCache(cfg.num_hidden_layers, 8, gm.nkv, gm.d, gm.dtype, gm.device), max_batch=4, max_seq_tokens=64, max_prefill_tokens=64)
    r.prefill([PrefillItem([1, 2, 3], 0, [1])])
    r.install([r.state.take_row(0)], [4], [3], [[1]], [1])
    r.resort()
    r.decode()                                   # (captures)
    on = torch.cuda.graph.default_capture_stream
    a = torch.zeros(8, device="cuda")
    for i in range(40):
        m = AdapterManager(gm, arena_bytes=1 << 20, host_bytes=1 << 20, max_slots=4)
        assert m.copy_stream.cuda_stream != on.cuda_stream, i
        if i % 8 == 0:
            size = 3000 + 4096 * i
            block = torch.zeros(size, dtype=torch.uint8).pin_memory()
            with torch.cuda.stream(m.copy_stream):
                block.to("cuda", non_blocking=True)
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, capture_error_mode="thread_local"):
                a.add_(1)
                del block
            for _ in range(2):
                torch.zeros(size, dtype=torch.uint8).pin_memory()


def test_engine_generate_runs_with_graphs():
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, cfg.vocab_size, (30 + i,), generator=g).tolist() for i in range(6)]
    eng = Engine(gm, EngineConfig(max_total_tokens=256, max_batch_prefill_tokens=1024), num_blocks=128, max_batch=8, use_graphs=True)
    a = eng.generate(prompts, max_new_tokens=16, adapter_indices=[0, 1, 2, 3, 1, 0])
    eng2 = Engine(gm, EngineConfig(max_total_tokens=256, max_batch_prefill_tokens=1024), num_blocks=128, max_batch=8, use_graphs=False)
    b = eng2.generate(prompts, max_new_tokens=16, adapter_indices=[0, 1, 2, 3, 1, 0])
    assert a == b          # graph replay and eager launches run the same kernels on the same data
    assert all(len(x) == 16 for x in a)


def test_smoke_entry():
    import __graft_entry__ as ge
    ge.smoke()


def test_mixtral_moe_gpu_matches_cpu_oracle():
    """Top-2 mixture of experts on the GPU kernels (dense form for decode-sized batches, gathered form for long prompts)
    against the fp32 CPU oracle of the same random model."""
    from lorax_b200.config import ModelConfig
    cfg = ModelConfig(model_type="mixtral", vocab_size=512, hidden_size=256, intermediate_size=384, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=64, rope_theta=1e4, max_position_embeddings=1024,
                      num_local_experts=4, num_experts_per_tok=2, torch_dtype="bfloat16")
    gm = DecoderModel.random_init(cfg, "cuda", torch.bfloat16, seed=2, std=0.05)
    cm = DecoderModel.random_init(cfg, "cpu", torch.float32, seed=2, std=0.05)
    g = torch.Generator().manual_seed(9)
    for n in (40, 300):                       # below / above the dense-form limit of 256 tokens
        prompt = torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist()
        outs = []
        for m in (gm, cm):
            kv = KVCache(cfg.num_hidden_layers, 32, m.nkv, m.d, m.dtype, m.device)
            r = ModelRunner(m, kv, max_batch=2, max_seq_tokens=512, max_prefill_tokens=512, use_graphs=False)
            _, _, logits = r.prefill([PrefillItem(prompt, 0, list(range(1, 12)), adapter_index=0)])
            outs.append(logits.float().cpu())
        err = ((outs[0] - outs[1]).norm() / outs[1].norm()).item()
        assert err < 4e-2, (n, err)
    from lorax_b200.ops import native
    native.workspace().check_status()


@pytest.mark.parametrize("family", ["bloom", "opt"])
def test_alibi_and_learned_position_families_match_cpu_oracle(family):
    """BLOOM (ALiBi, embedding LayerNorm, ungated GELU MLP) and OPT (learned positions with an offset, ReLU): prefill logits
    and teacher-forced decode logits on the GPU kernels against the fp32 CPU path of the same weights."""
    from lorax_b200.config import ModelConfig
    if family == "bloom":
        cfg = ModelConfig.from_dict({"model_type": "bloom", "vocab_size": 1000, "hidden_size": 256, "n_layer": 2, "n_head": 4,
                                     "layer_norm_epsilon": 1e-5, "seq_length": 512})
    else:
        cfg = ModelConfig.from_dict({"model_type": "opt", "vocab_size": 1000, "hidden_size": 256, "ffn_dim": 512, "num_hidden_layers": 2,
                                     "num_attention_heads": 4, "max_position_embeddings": 512, "word_embed_proj_dim": 256})
    gm = DecoderModel.random_init(cfg, "cuda", torch.bfloat16, seed=4, std=0.05)
    cm = DecoderModel.random_init(cfg, "cpu", torch.float32, seed=4, std=0.05)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (40, 75)]
    forced = torch.randint(0, cfg.vocab_size, (2,), generator=g).tolist()
    outs = []
    for m in (gm, cm):
        kv = KVCache(cfg.num_hidden_layers, 32, m.nkv, m.d, m.dtype, m.device)
        r = ModelRunner(m, kv, max_batch=4, max_seq_tokens=256, max_prefill_tokens=512, use_graphs=False)
        blocks = [[1, 2, 3, 4], [5, 6, 7, 8]]
        _, _, logits = r.prefill([PrefillItem(p, 0, b) for p, b in zip(prompts, blocks)])
        # one more token per sequence through the cached-context path
        _, _, step = r.prefill([PrefillItem([t], len(p), b) for t, p, b in zip(forced, prompts, blocks)])
        outs.append(torch.cat([logits.float().cpu(), step.float().cpu()]))
    from lorax_b200.ops import native
    native.workspace().check_status()
    err = (outs[0] - outs[1]).norm() / outs[1].norm()
    assert err < 3e-2, err


def test_engine_device_sampling_with_graphs():
    """Sampling rows inside graph-replayed decode steps: tokens depend on the request's seed only, greedy neighbours keep the
    tokens they have without any sampling request in the batch."""
    from lorax_b200.runtime.engine import GenRequest
    from lorax_b200.sampling.chooser import NextTokenParams
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    g = torch.Generator().manual_seed(31)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (9, 40, 17, 25)]
    sample = NextTokenParams(temperature=1.2, top_k=40, top_p=0.9, do_sample=True, seed=7)
    params = {0: NextTokenParams(), 1: sample, 2: NextTokenParams(temperature=0.7, typical_p=0.8, do_sample=True, seed=3), 3: NextTokenParams()}

    def run(order):
        eng = Engine(gm, EngineConfig(max_input_length=64, max_total_tokens=128, max_batch_prefill_tokens=256, compile=True), num_blocks=64)
        for rid in order:
            eng.add_request(GenRequest(rid, prompts[rid], max_new_tokens=12, params=params[rid], adapter_index=rid % 3))
        eng.run()
        return {rid: eng.finished[rid].output_ids for rid in order}
    a, b, greedy = run([0, 1, 2, 3]), run([2, 3, 1]), run([0, 3])
    assert a[1] == b[1] and a[2] == b[2] and a[3] == b[3] == greedy[3] and a[0] == greedy[0]
    assert all(len(v) == 12 for v in a.values())
    from lorax_b200.ops import native
    native.workspace().check_status()


def test_engine_device_penalties_with_graphs():
    """History penalties inside graph-replayed decode steps: the token histograms live on the device and are bumped in the step.
    A presence penalty far above the logits' range forbids every token already seen, so a greedy request's output neither
    repeats itself nor its prompt; the result does not depend on the batch around it, and a sampling request with penalties is
    reproducible from its seed."""
    from lorax_b200.runtime.engine import GenRequest
    from lorax_b200.sampling.chooser import NextTokenParams
    cfg, gm, _ = _build("cuda", torch.bfloat16)
    g = torch.Generator().manual_seed(37)
    prompts = [torch.randint(0, 60, (n,), generator=g).tolist() for n in (12, 33, 20)]
    params = {0: NextTokenParams(presence_penalty=1e4), 1: NextTokenParams(),
              2: NextTokenParams(temperature=0.9, top_k=30, do_sample=True, seed=5, repetition_penalty=1.4, frequency_penalty=0.3)}

    def run(order):
        eng = Engine(gm, EngineConfig(max_input_length=64, max_total_tokens=128, max_batch_prefill_tokens=256, compile=True), num_blocks=64)
        for rid in order:
            eng.add_request(GenRequest(rid, prompts[rid], max_new_tokens=16, params=params[rid], adapter_index=rid % 3))
        eng.run()
        assert not eng._hist
        return {rid: eng.finished[rid].output_ids for rid in order}
    a, b, greedy = run([0, 1, 2]), run([2, 0]), run([1])
    assert len(set(a[0])) == 16 and not set(a[0]) & set(prompts[0])
    assert a[0] == b[0] and a[2] == b[2] and a[1] == greedy[1]
    from lorax_b200.ops import native
    native.workspace().check_status()


_FAMILY_CONFIGS = {
    "gemma2": {"model_type": "gemma2", "num_key_value_heads": 2, "head_dim": 64, "sliding_window": 32, "query_pre_attn_scalar": 64,
               "attn_logit_softcapping": 30.0, "final_logit_softcapping": 20.0, "rms_norm_eps": 1e-6},
    "phi3": {"model_type": "phi3", "num_key_value_heads": 2},
    "gpt_neox": {"model_type": "gpt_neox", "rotary_pct": 0.25, "use_parallel_residual": True, "layer_norm_eps": 1e-5},
    "falcon": {"model_type": "falcon", "multi_query": True, "parallel_attn": True, "bias": False, "new_decoder_architecture": False},
    "cohere": {"model_type": "cohere", "num_key_value_heads": 2, "logit_scale": 0.25, "layer_norm_eps": 1e-5},
    "granite": {"model_type": "granite", "num_key_value_heads": 2, "embedding_multiplier": 3.0, "logits_scaling": 2.0,
                "residual_multiplier": 0.5, "attention_multiplier": 0.1},
    "gpt2": {"model_type": "gpt2", "n_embd": 256, "n_layer": 2, "n_head": 4, "n_positions": 512},
    "phi": {"model_type": "phi", "partial_rotary_factor": 0.5, "layer_norm_eps": 1e-5},
    "mistral_window": {"model_type": "mistral", "num_key_value_heads": 2, "sliding_window": 32},
}


@pytest.mark.parametrize("family", sorted(_FAMILY_CONFIGS))
def test_decoder_families_match_cpu_oracle(family):
    """The architecture switches of the config-driven decoder on the GPU kernels (soft caps and alternating windows of gemma2,
    partial rotary and parallel residuals of neox / phi / falcon, multi-query attention, bias-free LayerNorm of cohere, the
    multipliers of granite, learned positions of gpt2, a sliding window shorter than the prompt): prefill logits and
    teacher-forced decode logits against the fp32 CPU path of the same random weights."""
    from lorax_b200.config import ModelConfig
    d = {"vocab_size": 1000, "hidden_size": 256, "intermediate_size": 512, "num_hidden_layers": 2, "num_attention_heads": 4,
         "max_position_embeddings": 512}
    d.update(_FAMILY_CONFIGS[family])
    cfg = ModelConfig.from_dict(d)
    gm = DecoderModel.random_init(cfg, "cuda", torch.bfloat16, seed=4, std=0.05)
    cm = DecoderModel.random_init(cfg, "cpu", torch.float32, seed=4, std=0.05)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (40, 75)]
    forced = torch.randint(0, cfg.vocab_size, (2,), generator=g).tolist()
    outs = []
    for m in (gm, cm):
        kv = KVCache(cfg.num_hidden_layers, 32, m.nkv, m.d, m.dtype, m.device)
        r = ModelRunner(m, kv, max_batch=4, max_seq_tokens=256, max_prefill_tokens=512, use_graphs=False)
        blocks = [[1, 2, 3, 4], [5, 6, 7, 8]]
        _, _, logits = r.prefill([PrefillItem(p, 0, b) for p, b in zip(prompts, blocks)])
        _, _, step = r.prefill([PrefillItem([t], len(p), b) for t, p, b in zip(forced, prompts, blocks)])
        outs.append(torch.cat([logits.float().cpu(), step.float().cpu()]))
    from lorax_b200.ops import native
    native.workspace().check_status()
    err = (outs[0] - outs[1]).norm() / outs[1].norm()
    assert err < 3e-2, err
