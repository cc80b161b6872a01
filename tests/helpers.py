"""Shared builders for the test-suite: tiny seeded models and compressors."""
import ctypes
import os
import re
import tempfile

import torch

from fastcache_b200.config import ModelConfig


def tiny_llama_config(**over):
    cfg = dict(model_type="llama", architectures=["LlamaForCausalLM"], hidden_size=256,
               num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64,
               intermediate_size=512, vocab_size=1024, rope_theta=10000.0, rms_norm_eps=1e-6,
               max_position_embeddings=2048, tie_word_embeddings=False, eos_token_id=2)
    cfg.update(over)
    return ModelConfig(**cfg)


def tiny_qwen3_config(**over):
    return tiny_llama_config(model_type="qwen3", architectures=["Qwen3ForCausalLM"], **over)


def random_compressor(cls, n_layer, head_dim, factor, seed=0, **kw):
    torch.manual_seed(seed)
    m = cls(None, factor, kw.pop("min_seq_len", 1), n_layer=n_layer, nhead=2, head_dim=head_dim)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    return m.eval()


def _demangled(name):
    lib = ctypes.CDLL("libstdc++.so.6")
    lib.__cxa_demangle.restype = ctypes.c_char_p
    status = ctypes.c_int()
    plain = lib.__cxa_demangle(name.encode(), None, None, ctypes.byref(status))
    return plain.decode() if status.value == 0 else name


def launched(f, *parts):
    """Names (demangled, without blanks) of the kernels that f() launches and that hold one of `parts`, read from a capture."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.stream(stream):
        f()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            f()
    with tempfile.TemporaryDirectory() as folder:
        path = os.path.join(folder, "graph.dot")
        assert ctypes.CDLL("libcuda.so.1").cuGraphDebugDotPrint(ctypes.c_void_p(graph.raw_cuda_graph()), path.encode(), 1) == 0
        with open(path) as dot:
            names = {_demangled(n).replace(" ", "") for n in re.findall(r"_ZN?[A-Za-z0-9_]+", dot.read())}
    return sorted(n for n in names if any(p in n for p in parts))
