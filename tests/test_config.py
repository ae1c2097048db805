"""Configuration and registry (no GPU): every size comes from config.json; what the engine
cannot honour is refused with the key's name (model/config.go:132-312, model/model.go:95-192)."""
import copy

import pytest

import tiny
from tgo_b200.config.qwen3 import ConfigError, Qwen3Config, qwen3_model_spec
from tgo_b200.registry import ARCHITECTURES, Registry, model_spec_from_config


def test_tiny_configs_differ_in_every_size_and_option():
    a, b = Qwen3Config.from_dict(tiny.TINY_A), Qwen3Config.from_dict(tiny.TINY_B)
    for f in ("hidden_size", "num_hidden_layers", "num_attention_heads", "head_dim",
              "intermediate_size", "vocab_size", "rms_norm_eps", "rope_theta",
              "tie_word_embeddings", "max_position_embeddings", "kv_group", "q_width"):
        assert getattr(a, f) != getattr(b, f), f
    assert a.layer_windows == (None, None) and b.layer_windows == (None, 24, None)
    assert b.q_width != b.hidden_size          # head_dim from the file, not hidden/heads
    assert tiny.TINY_A_RUN["page_size"] != tiny.TINY_B_RUN["page_size"]


def test_spec_carries_the_files_numbers():
    spec = qwen3_model_spec(tiny.TINY_B)
    assert spec.architecture == "Qwen3ForCausalLM" and spec.hidden_size == 96
    assert len(spec.layers) == 3 and [c.layer for c in spec.run_order] == [0, 1, 2]
    m = spec.layers[1].mixer
    assert (m.num_heads, m.num_kv_heads, m.head_dim, m.window, m.qk_norm) == (6, 2, 32, 24, True)
    assert m.position.theta == 1e6 and m.position.rotary_dim == 32 and m.norm_eps == 1e-5
    assert spec.layers[0].mixer.window is None
    assert spec.layers[2].feed_forward.intermediate_size == 224
    assert spec.head_name == "lm_head.weight" and spec.tied_head_alias is None
    tied = qwen3_model_spec(tiny.TINY_A)
    assert tied.head_name is None and tied.tied_head_alias == "lm_head.weight"


def test_defaults_head_dim_and_kv_heads():
    raw = copy.deepcopy(tiny.TINY_A)
    del raw["head_dim"], raw["num_key_value_heads"]
    c = Qwen3Config.from_dict(raw)
    assert c.head_dim == 16 and c.num_key_value_heads == 4


@pytest.mark.parametrize("edit,needle", [
    (lambda r: r.pop("hidden_size"), "hidden_size is required"),
    (lambda r: r.update(num_hidden_layers=0), "num_hidden_layers is 0"),
    (lambda r: r.update(vocab_size=-3), "vocab_size"),
    (lambda r: r.pop("rms_norm_eps"), "rms_norm_eps is required"),
    (lambda r: r.update(rope_theta=1e60), "rope_theta"),
    (lambda r: r.update(rms_norm_eps=1e-60), "rms_norm_eps"),
    (lambda r: r.update(head_dim=15), "head_dim is 15"),
    (lambda r: r.update(num_key_value_heads=3), "num_key_value_heads"),
    (lambda r: r.update(rope_scaling={"rope_type": "yarn", "factor": 4}), "rope_scaling is set (yarn)"),
    (lambda r: r.update(attention_bias=True), "attention_bias"),
    (lambda r: r.update(hidden_act="gelu"), "hidden_act"),
    (lambda r: r.update(sliding_window=64, use_sliding_window=None) or r.pop("use_sliding_window"),
     "sliding_window is 64"),
    (lambda r: r.update(use_sliding_window=True, sliding_window=None), "use_sliding_window"),
    (lambda r: r.update(layer_types=["full_attention"]), "layer_types"),
    (lambda r: r.update(layer_types=["full_attention", "sliding_attention"], sliding_window=None),
     "sliding_window is not set"),
    (lambda r: r.update(layer_types=["full_attention", "linear_attention"]), "known kinds"),
    (lambda r: r.update(max_position_embeddings=None), "max_position_embeddings is required"),
    (lambda r: r.update(architectures=[]), "architectures[0]"),
])
def test_refusals_name_the_key(edit, needle):
    raw = copy.deepcopy(tiny.TINY_A)
    edit(raw)
    with pytest.raises(ConfigError) as e:
        Qwen3Config.from_dict(raw)
    assert needle in str(e.value)


def test_head_dim_default_must_divide():
    raw = copy.deepcopy(tiny.TINY_A)
    del raw["head_dim"]
    raw["num_attention_heads"] = 6
    raw["num_key_value_heads"] = 2
    with pytest.raises(ConfigError, match="head_dim is absent"):
        Qwen3Config.from_dict(raw)


def test_use_sliding_window_with_max_window_layers():
    raw = copy.deepcopy(tiny.TINY_B)
    del raw["layer_types"]
    raw.update(use_sliding_window=True, max_window_layers=2, sliding_window=10)
    assert Qwen3Config.from_dict(raw).layer_windows == (None, None, 10)


def test_null_rope_scaling_and_qwen_window_keys_pass():
    raw = dict(tiny.TINY_A, rope_scaling=None, sliding_window=None, use_sliding_window=False)
    assert Qwen3Config.from_dict(raw).layer_windows == (None, None)


def test_registry_unknown_lists_known_and_duplicates_raise():
    with pytest.raises(KeyError) as e:
        model_spec_from_config({"architectures": ["NoSuchModel"]})
    assert "Qwen3ForCausalLM" in str(e.value) and "NoSuchModel" in str(e.value)
    r = Registry("thing")
    r.register("a", object)
    with pytest.raises(ValueError, match="twice"):
        r.register("a", object)
    with pytest.raises(ValueError, match="needs a name"):
        r.register("", object)
    with pytest.raises(ValueError, match="no constructor"):
        r.register("b", None)
    assert "Qwen3ForCausalLM" in ARCHITECTURES.names()


def test_run_order_is_validated():
    from tgo_b200.config.spec import LayerCall
    spec = qwen3_model_spec(tiny.TINY_A)
    spec.run_order = [LayerCall(0), LayerCall(5)]
    with pytest.raises(ValueError, match="names layer 5"):
        spec.validate()
    spec.run_order = [LayerCall(0, cache_from=0)]
    with pytest.raises(ValueError, match="does not run before"):
        spec.validate()
    spec.run_order = [LayerCall(0), LayerCall(1, cache_from=0), LayerCall(0, cache_from=1)]
    with pytest.raises(ValueError, match="owns none"):
        spec.validate()
    spec.run_order = [LayerCall(0), LayerCall(1), LayerCall(0, cache_from=0)]
    spec.validate()


def test_build_folder_is_one_for_all_threads():
    """Several libraries compile side by side: every thread must get the same folder (a
    probe file shared by name once sent some of them to the fallback folder)."""
    from concurrent.futures import ThreadPoolExecutor

    from tgo_b200.kernels import build as kb
    kb._build_dir_found = None
    with ThreadPoolExecutor(max_workers=8) as pool:
        got = set(pool.map(lambda _: kb._build_dir(), range(64)))
    assert len(got) == 1
    # and the host library, which needs no CUDA compiler, builds and loads
    lib = kb.load_library("host_runtime")
    assert lib.tgo_cache_create


def test_entry_points_hand_over_what_ctypes_does(tmp_path):
    """Whole numbers of every width, singles and doubles in any order and number, against ctypes."""
    import ctypes
    import subprocess

    from tgo_b200.kernels import build as kb
    if kb.find_host_compiler() is None:
        pytest.skip("no host compiler")
    src = tmp_path / "probe.cpp"
    src.write_text("""
extern "C" int many(int a, float b, long long c, double d, const void* e, short f, int g, int h, float i, long long j,
                    int k, int l, int m, int n, float o, const void* p) {
    return (a == -1) + 2 * (b == 0.1f) + 4 * (c == -(1ll << 40)) + 8 * (d == 0.1) + 16 * (e == (void*)0xffff800000000010ull) +
           32 * (f == -7) + 64 * (g == 5) + 128 * (h == 1) + 256 * (i == -2.5f) + 512 * (j == (1ll << 62)) + 1024 * (k == 0) +
           2048 * (l == 11) + 4096 * (m == 12) + 8192 * (n == -13) + 16384 * (o == 3.0f) + 32768 * (p == 0);
}
extern "C" int negative() { return -3; }
""")
    so = tmp_path / "probe.so"
    subprocess.run([kb.find_host_compiler(), "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    args = (-1, 0.1, -(1 << 40), (0.1,), 0xffff800000000010, -7, 5, True, -2.5, 1 << 62, 0, 11, 12, -13, 3.0, 0)
    for bind in (kb._find_binder(), kb._bind_ctypes):
        entries = kb._Entries(lib, bind)
        assert entries.many(*args) == 65535 and entries.negative() == -3
    fast = kb._Entries(lib, kb._find_binder()).many
    if kb._find_binder() is not kb._bind_ctypes:
        for bad in ("x", None, b"y", (1.0, 2.0), 1 << 70):
            with pytest.raises((TypeError, OverflowError)):
                fast(bad)
        with pytest.raises(TypeError):
            fast(*([0] * 49))


def test_kernels_are_called_by_ctypes_where_the_extension_fails(monkeypatch, tmp_path, capfd):
    """The extension that calls the kernels does not compile, or what was built does not load: ctypes calls
    them, and building everything goes on. A library of kernels that fails still raises."""
    from tgo_b200.kernels import build as kb
    broken = tmp_path / "broken.so"
    broken.write_bytes(b"no library")

    def fails(name, **kw):
        raise kb.KernelBuildError(f"the compiler failed on {name}")
    for compiles in (fails, lambda name, **kw: str(broken)):
        monkeypatch.setattr(kb, "compile_library", compiles)
        assert kb._find_binder() is kb._bind_ctypes
        assert "ctypes" in capfd.readouterr().err
    monkeypatch.setattr(kb, "compile_library", lambda name, verbose=True: fails(name))
    monkeypatch.setattr(kb, "library_path", lambda name: str(tmp_path / name))
    monkeypatch.setattr(kb, "LIBRARIES", {"fastcall": kb.LIBRARIES["fastcall"]})
    kb.build_all(verbose=False)
    monkeypatch.setattr(kb, "LIBRARIES", {"fastcall": ([], []), "other": ([], []), "third": ([], [])})
    with pytest.raises(kb.KernelBuildError, match="other|third"):
        kb.build_all(verbose=False)


def test_python_extension_is_built_for_each_interpreter(monkeypatch, tmp_path):
    """A build folder shared by interpreters of unlike binary interfaces holds an extension for each, and
    building one leaves the other's."""
    from tgo_b200.kernels import build as kb
    if kb.find_host_compiler() is None or kb._find_binder() is kb._bind_ctypes:
        pytest.skip("no extension here")
    monkeypatch.setattr(kb, "_build_dir_found", str(tmp_path))
    mine, books = kb.library_path("fastcall"), kb.library_path("host_runtime")
    with monkeypatch.context() as m:
        m.setattr(kb.sysconfig, "get_config_var", lambda name: "cpython-399td-x86_64-linux-gnu")
        other = kb.library_path("fastcall")
        assert kb.library_path("host_runtime") == books
    assert other != mine
    with open(other, "w") as f:
        f.write("another interpreter's")
    assert kb.compile_library("fastcall", verbose=False) == mine
    import os
    assert os.path.exists(other) and os.path.exists(mine)


def test_engine_compiles_all_it_calls_at_once(monkeypatch):
    """Everything an engine on a GPU will load is compiled when it is made, side by side: the libraries its
    model names, the books, and what calls the kernels."""
    import types

    import torch
    from tgo_b200.engine import step
    asked = []
    monkeypatch.setattr(step, "compile_together", lambda names, **kw: asked.extend(names))
    monkeypatch.setattr(step, "NativeCacheManager", lambda *a: None)
    monkeypatch.setattr(step, "CacheStorage", lambda *a: None)
    model = types.SimpleNamespace(device=torch.device("cuda"), groups=[], dtype=torch.bfloat16, state_shapes=[],
                                  libraries=lambda page_size: ["moe", "gemm_tc"])
    step.Engine(model, max_tokens=64)
    assert {"host_runtime", "fastcall", "moe", "gemm_tc"} <= set(asked)


@pytest.mark.parametrize("which", ["grouped", "latent"])
def test_counters_live_until_the_launch(which, monkeypatch):
    """The counters a launch draws its items from are still held when the launch is made: memory that went
    back to the allocator before it may be another thread's by then."""
    import gc
    import types
    import weakref

    import torch
    from tgo_b200.kernels import ops
    made, launched = [], []
    empty = torch.empty

    def recorded(*a, **kw):
        t = empty(*a, **kw)
        made.append(weakref.ref(t))
        return t

    def launch(*args):
        gc.collect()
        launched.append([r() is not None and r().data_ptr() in args for r in made])
        return 0
    fake = types.SimpleNamespace(tgo_attention_tc_prefill=launch, tgo_attention_latent_tc=launch)
    for name, value in (("_need_cuda", lambda *a: None), ("_stream", lambda: 0), ("entry_points", lambda name: fake)):
        monkeypatch.setattr(ops, name, value)
    i32 = torch.zeros(4, dtype=torch.int32)
    q, out = torch.zeros(4, 256, dtype=torch.bfloat16), torch.zeros(4, 256, dtype=torch.bfloat16)
    cache = torch.zeros(3, 1, 16, 128, dtype=torch.bfloat16)
    monkeypatch.setattr(torch, "empty", recorded)
    if which == "grouped":
        ops.attention_tc_prefill(q, out, 2, 1, 128, cache, cache, 16, i32.view(2, 2), i32, i32, i32, i32, 0.1, 0,
                                 own_counters=True)
    else:
        ops.attention_latent_tc(q, out, 2, 128, 64, cache, 16, i32.view(2, 2), i32, i32, 0.1, 0, None, i32, i32)
    assert launched == [[True]]


def test_chunked_scan_refuses_a_short_workspace():
    """The library says how long a chunk is, and a workspace of one float less than its chunks need for one
    head is refused before anything is launched (the addresses below are never read)."""
    from tgo_b200.kernels import ops
    from tgo_b200.kernels.build import entry_points
    lib = entry_points("state_space")
    T, B, H, G, N, P = 300, 3, 4, 2, 128, 64
    chunk = lib.tgo_ssd_chunk_tokens()
    floats = (T // chunk + B) * (N * P + 3 * chunk + 4)
    at = 1 << 20
    for short in (floats - 1, 0, -1):
        assert lib.tgo_ssd_scan(at, H * P + 2 * G * N, at, H, 0, at, 0, at, T, B, H, G, N, P, at, at, at, H * N * P, 0, at,
                                short, 0) == ops.E_BAD_ARG


@pytest.mark.parametrize("N,K,E,top,tokens", [(1536, 4096, 16, 2, (8, 16, 33, 64)), (768, 4096, 128, 8, (4,))])
def test_routed_products_stay_off_the_narrowest_tiles(N, K, E, top, tokens):
    """Decode batches for which tiles of 32 gated columns were slower than all wider ones (and than the
    kernels before them): 108 us against 68 to 81 at the first, 173 against 85 to 98 at the fourth."""
    from tgo_b200.kernels.build import entry_points
    for T in tokens:
        assert entry_points("moe").tgo_moe_tile_width(N, K, E, T * top, 1, 148) >= 64


def test_selective_scan_of_no_requests_at_all(monkeypatch):
    """A step without requests launches what does nothing; the rule for chunks does not divide by their count."""
    import types

    import torch
    from tgo_b200.kernels import ops
    seen = []
    lib = types.SimpleNamespace(tgo_ssd_chunk_tokens=lambda: 64, tgo_selective_scan=lambda *a: seen.append(a) or 0)
    for name, value in (("_need_cuda", lambda *a: None), ("_stream", lambda: 0), ("entry_points", lambda name: lib)):
        monkeypatch.setattr(ops, name, value)
    z = torch.zeros
    ops.selective_scan(z(0, 2 * 64 + 2 * 64), z(0, 2, dtype=torch.bfloat16), None, z(2), None, z(0, 128), 0, 2, 1, 64, 64,
                       z(1, dtype=torch.int32), z(0, dtype=torch.int32), z(1, 2 * 64 * 64), 0)
    assert len(seen) == 1
