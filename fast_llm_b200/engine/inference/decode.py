"""Native generation steps: one new position per row of an attention decoder in one host call (`csrc/decode.cu`).

`DecodePlan.build(model)` describes the decoder to the kernels, or returns None when some part of it is not theirs (mixture of
experts, adapters, per-head norms, tensor parallelism, ...): those models step through their layers.
"""

import ctypes

import torch

from fast_llm_b200.layers.attention import Attention
from fast_llm_b200.layers.block import DecoderBlock
from fast_llm_b200.layers.language_model import LanguageModelEmbedding, LanguageModelHead
from fast_llm_b200.layers.linear import LinearBase
from fast_llm_b200.layers.mlp import MLP
from fast_llm_b200.layers.normalization import FixedRMSNormalization, LayerNormalization, RMSNormalization
from fast_llm_b200.layers.rotary import DefaultRotary, Llama3Rotary, NoRotary, ProportionalRotary, YarnRotary
from fast_llm_b200.ops import _lib

MAX_ROWS = 32
_NORM_KINDS = {RMSNormalization: 1, FixedRMSNormalization: 1, LayerNormalization: 2}
_ZERO_CENTERED = 4


class _Layer(ctypes.Structure):
    _fields_ = ([(name, ctypes.c_void_p) for name in ("norm1_w", "norm1_b", "qkv_w", "qkv_b", "dense_w", "dense_b", "norm2_w", "norm2_b", "w1", "b1",
                                                      "w2", "b2", "table")]
                + [(name, ctypes.c_int) for name in ("norm1", "norm2", "heads", "kv_heads", "head_dim", "rot_dim", "window", "ffn", "gated", "act")]
                + [(name, ctypes.c_float) for name in ("eps1", "eps2", "scale")])


class _Unsupported(Exception):
    pass


def _require(condition) -> None:
    if not condition:
        raise _Unsupported


def _weight(tensor) -> int:
    _require(torch.is_tensor(tensor) and tensor.is_cuda and tensor.dtype == torch.bfloat16 and tensor.is_contiguous() and tensor.data_ptr() % 16 == 0)
    return tensor.data_ptr()


def _norm(layer) -> tuple[int | None, int | None, int, float]:
    _require(type(layer) in _NORM_KINDS)
    kind = _NORM_KINDS[type(layer)] | (_ZERO_CENTERED if getattr(layer._config, "zero_centered", False) else 0)
    return (_weight(layer.weight) if layer.has_weight else None, _weight(layer.bias) if type(layer) is LayerNormalization else None, kind,
            layer._config.epsilon)


def _linear(layer) -> tuple[int, int | None]:
    _require(isinstance(layer, LinearBase) and layer._forward_hook is None and layer._group is None)
    return _weight(layer.weight), _weight(layer.bias) if layer._has_bias else None


class DecodePlan:
    def __init__(self, model):
        layers = [layer.unwrap() for layer in model.base_model.get_layers()]
        _require(len(layers) >= 3 and type(layers[0]) is LanguageModelEmbedding and type(layers[-1]) is LanguageModelHead
                 and all(type(layer) is DecoderBlock for layer in layers[1:-1]))
        # stages that share weight buffers re-fill them between stages: no fixed addresses
        _require(model._num_weight_buffers == len(model.stages_on_device) == len(model.stages))
        embedding, head = layers[0], layers[-1]
        _require(not embedding._has_position_embeddings and embedding._tp_dim.size == 1 and embedding._residual_dtype == torch.bfloat16)
        self._stages = list(model.stages_on_device.values())
        self._hidden, self._vocab = embedding._hidden_dim.size, head._vocab_size
        self._embedding, self._embedding_scale = _weight(embedding.word_embeddings_weight), float(embedding._config.embedding_scale)
        _require(head._logits_group is None)
        self._final = _norm(head.final_norm)
        self._head_config, self._head = head._config, _weight(head.output_weights)
        self._rotary, self._layers = [], (_Layer * (len(layers) - 2))()
        for out, block in zip(self._layers, layers[1:-1]):
            self._describe(block, out)
        self._cache_width = 2 * self._layers[0].kv_heads * self._layers[0].head_dim
        _require(all(2 * l.kv_heads * l.head_dim == self._cache_width for l in self._layers))
        self._supported = [bool(_lib.get_lib().flb_decode_supported(self._layers, len(self._layers), self._hidden, rows)) for rows in range(MAX_ROWS + 1)]

    def _describe(self, block, out: _Layer) -> None:
        c, mixer, mlp = block._config, block.mixer, block.mlp
        _require(not block._return_input and c.post_mixer_normalization is None and c.post_mlp_normalization is None and not block._has_output_scale
                 and type(mixer) is Attention and type(mlp) is MLP)
        a, m = mixer._config, mlp._config
        _require(not mixer._has_head_norms and not a.shared_key_value and a.causal and mixer._sdp_dim.size == 1)
        (q, q_bias), (kv, kv_bias) = _linear(mixer.query), _linear(mixer.key_value)
        _require(q + mixer.query.weight.numel() * 2 == kv)
        _require((q_bias is None) == (kv_bias is None) and (q_bias is None or q_bias + mixer.query.bias.numel() * 2 == kv_bias))
        _require(m.pre_norm is None and m.post_norm is None and not mlp.layer_1.transposed_weight and mlp.layer_2.transposed_weight)
        out.norm1_w, out.norm1_b, out.norm1, out.eps1 = _norm(block.norm_1)
        out.norm2_w, out.norm2_b, out.norm2, out.eps2 = _norm(block.norm_2)
        out.qkv_w, out.qkv_b = q, q_bias
        out.dense_w, out.dense_b = _linear(mixer.dense)
        out.w1, out.b1 = _linear(mlp.layer_1)
        out.w2, out.b2 = _linear(mlp.layer_2)
        out.heads, out.kv_heads, out.head_dim, out.window = mixer._local_heads, mixer._local_head_groups, a.head_size, a.window_size or 0
        out.scale, out.ffn, out.gated, out.act = mixer._softmax_scale, m.intermediate_size, int(m.gated), m.activation.code
        rotary = mixer._rotary
        _require(type(rotary) in (NoRotary, DefaultRotary, Llama3Rotary, YarnRotary, ProportionalRotary))
        out.rot_dim = 0 if type(rotary) is NoRotary else rotary.rot_dim
        self._rotary.append(None if out.rot_dim == 0 else rotary)

    @classmethod
    def build(cls, model) -> "DecodePlan | None":
        if model.distributed.device.type != "cuda":
            return None
        try:
            return cls(model)
        except (_Unsupported, AttributeError):
            return None

    def takes(self, rows: int, new: int, cache) -> bool:
        return new == 1 and cache.length > 0 and rows <= MAX_ROWS and self._supported[rows] and cache.width in (None, self._cache_width)

    @torch.no_grad()
    def step(self, tokens: torch.Tensor, cache, device) -> torch.Tensor:
        """tokens [rows, 1]: the next position of every row of `cache`.  Returns logits [rows, vocab] and extends the cache."""
        for stage in self._stages:
            stage.restore_parameters()
        rows, length = tokens.shape[0], cache.length
        # this call's own copy: another thread may step the same model
        layers = type(self._layers).from_buffer_copy(self._layers)
        tables = [None if rotary is None else rotary.get_table(length + 2, device) for rotary in self._rotary]
        for layer, table in zip(layers, tables):
            layer.table = _lib.ptr(table)
        ids = tokens.reshape(-1).to(device=device, dtype=torch.int64).contiguous()  # a column of a wider tensor stays strided otherwise
        buffer, pads = cache.reserve(length + 1, len(self._layers), self._cache_width, device)
        lib = _lib.get_lib()
        workspace = torch.empty(lib.flb_decode_workspace(layers, len(layers), self._hidden, rows), dtype=torch.uint8, device=device)
        logits = torch.empty(rows, self._vocab, dtype=torch.float32, device=device)
        final_w, final_b, final_norm, final_eps = self._final
        _lib.check(lib.flb_decode_step(
            layers, len(layers), ids.data_ptr(), rows, self._embedding, self._embedding_scale, self._hidden, self._vocab, final_w, final_b,
            final_norm, final_eps, self._head, buffer.data_ptr(), buffer.stride(0), buffer.shape[2], length, pads.data_ptr(),
            workspace.data_ptr(), logits.data_ptr(), _lib.stream_ptr()), "flb_decode_step")
        _lib.count_launch(9 * len(layers) + 4)
        cache.length = length + 1
        c = self._head_config
        if c.logits_scale_factor != 1.0:
            logits = logits * c.logits_scale_factor
        if c.final_logit_softcap is not None:
            logits = torch.tanh(logits / c.final_logit_softcap) * c.final_logit_softcap
        return logits
