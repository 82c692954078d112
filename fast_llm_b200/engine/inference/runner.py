"""Forward-only execution of a staged model (reference models for distillation / preference losses, evaluation,
generation).  Parity: `fast_llm/engine/inference/runner.py:13-71`."""

import torch

from fast_llm_b200.data.document import LanguageModelBatch, LanguageModelDocument
from fast_llm_b200.engine.multi_stage.config import StageMode
from fast_llm_b200.parallel.topology import PhaseType


class KeyValueCache:
    """Generation cache of an attention-only decoder.  Per attention layer, in layer order: the rotated keys and values of
    every row's positions so far, `[rows * length, width]` with the rows one after another (a row's left padding included:
    it is a document of its own, as in the packed forward pass).  Parity: the `past_key_values` / `presents` lists of
    `fast_llm/models/gpt/huggingface.py:158-199`.

    Generation steps append to one buffer `[layers, rows, capacity, width]` with room for more positions (an eighth, at least 256),
    so a step writes its own position instead of copying all earlier ones.  Where the memory does not have that room, the buffer
    is exactly as long as asked for."""

    def __init__(self, pads: list[int]):
        self.pads = list(pads)  # left padding of every row
        self.length = 0  # positions held per row
        self.on_reorder = None  # called with the row index before a reorder (tensor-parallel workers follow it)
        self._layers: list[torch.Tensor] = []
        self._buffer: torch.Tensor | None = None  # holds the positions instead of `_layers` once a step has reserved it
        self._device_pads: torch.Tensor | None = None

    @property
    def rows(self) -> int:
        return len(self.pads)

    @property
    def width(self) -> int | None:
        """Elements per position of a layer, None while empty or if the layers differ."""
        if self._buffer is not None:
            return self._buffer.shape[-1]
        widths = {t.shape[-1] for t in self._layers}
        return widths.pop() if len(widths) == 1 else None if not widths else -1

    @property
    def layers(self) -> list[torch.Tensor]:
        if self._buffer is not None:
            return [t[:, : self.length].reshape(self.rows * self.length, -1) for t in self._buffer.unbind(0)]
        return self._layers

    @layers.setter
    def layers(self, layers: list[torch.Tensor]) -> None:
        self._layers, self._buffer = list(layers), None

    def reserve(self, length: int, layers: int, width: int, device) -> tuple[torch.Tensor, torch.Tensor]:
        """(buffer with room for `length` positions of every row, left padding of the rows on the device)."""
        if self._buffer is None or self._buffer.shape[2] < length:
            def allocate(capacity):
                return torch.empty(layers, self.rows, capacity, width, dtype=torch.bfloat16, device=device)

            try:
                buffer = allocate(-(-(length + max(length // 8, 256)) // 64) * 64)
            except torch.cuda.OutOfMemoryError:
                buffer = allocate(length)
            if self._buffer is not None:
                buffer[:, :, : self.length] = self._buffer[:, :, : self.length]
            else:
                for i, kv in enumerate(self._layers):
                    buffer[i, :, : self.length] = kv.view(self.rows, self.length, width)
            buffer[:, :, self.length :] = 0  # masked keys are still multiplied: they have to be finite
            self._buffer, self._layers = buffer, []
        if self._device_pads is None:
            self._device_pads = torch.tensor(self.pads, dtype=torch.int32, device=device)
        return self._buffer, self._device_pads

    def __copy__(self) -> "KeyValueCache":
        """A branch of the generation: later steps of either cache do not show in the other."""
        other = KeyValueCache(self.pads)
        other.__dict__.update(self.__dict__)
        other.pads, other._layers = list(self.pads), list(self._layers)
        if self._buffer is not None:
            other._buffer = self._buffer.clone()
        return other

    def get_seq_length(self, layer_idx: int = 0) -> int:
        return self.length

    def reorder_cache(self, beam_idx: torch.Tensor) -> None:
        """The name `transformers` beam search calls."""
        if self.on_reorder is not None:
            self.on_reorder(beam_idx)
        self.reorder(beam_idx)

    def reorder(self, index: torch.Tensor) -> None:
        """Beam search: row i continues from row index[i]."""
        order = index.tolist()
        if self._buffer is not None:
            self._buffer = self._buffer.index_select(1, index.to(self._buffer.device))
        else:
            self._layers = [kv.view(self.rows, self.length, -1).index_select(0, index.to(kv.device)).reshape(len(order) * self.length, -1)
                            for kv in self._layers]
        self.pads = [self.pads[i] for i in order]
        self._device_pads = None


class InferenceRunner:
    def __init__(self, model):
        self._model = model
        self._is_setup = False
        self._plan: tuple | None = None

    @property
    def model(self):
        return self._model

    def setup(self, distributed=None, pretrained_config=None) -> None:
        if not self._model.is_setup:
            self._model.setup(distributed, mode=StageMode.inference)
        self._distributed = self._model.distributed
        self._is_setup = True

    def load(self, pretrained_config) -> None:
        if pretrained_config.pretrained.path is not None:
            self._model.load_checkpoint(pretrained_config.pretrained)
        else:
            self._model.initialize_weights()

    @torch.no_grad()
    def forward_kwargs(self, tokens: torch.Tensor, kwargs: dict, iteration: int = 0) -> dict:
        """Run every stage on one prepared micro-sequence; results (logits, hidden states) land in `kwargs`."""
        assert self._is_setup
        kwargs["training"] = False
        output = tokens
        for stage in self._model.stages_on_device.values():
            stage.restore_parameters()
            output, _ = stage.forward(output, kwargs)
        return kwargs

    @torch.no_grad()
    def forward_tokens(self, tokens: torch.Tensor, document_lengths: list[int] | None = None, output_hidden_states=None):
        """Logits [tokens, vocab] for a flat token stream (one document unless lengths are given).  With
        `output_hidden_states` (a list of layer names, possibly empty) returns `(logits, {name: hidden})`."""
        n = len(tokens)
        lengths = document_lengths or [n]
        batch = LanguageModelBatch(tokens=torch.cat([tokens.cpu().long(), torch.full((1,), -100, dtype=torch.long)]),
                                   document_lengths=lengths[:-1] + [lengths[-1] + 1])
        (inp,) = batch.get_model_inputs(micro_batch_size=n, predicted_tokens=1)
        kwargs = inp.to_kwargs(self._distributed.device)
        kwargs.pop("labels", None)
        kwargs["return_logits"] = True
        if output_hidden_states:
            kwargs["output_hidden_states"] = set(output_hidden_states)
            kwargs["hidden_states"] = {}
        for layer in self._model.base_model.get_layers():
            layer.preprocess(kwargs)
        self.forward_kwargs(kwargs["token_ids"], kwargs)
        if output_hidden_states is not None:
            return kwargs["logits"], kwargs.get("hidden_states", {})
        return kwargs["logits"]

    def supports_key_value_cache(self) -> bool:
        """True when every mixer of the decoder is attention on this rank's own sequence (recurrent mixers keep no state
        between calls, sequence-data parallelism splits the keys)."""
        from fast_llm_b200.layers.attention import Attention
        from fast_llm_b200.layers.block import DecoderBlock

        blocks = [layer.unwrap() for layer in self._model.base_model.get_layers() if isinstance(layer.unwrap(), DecoderBlock)]
        return bool(blocks) and all(type(block.mixer) is Attention and block.mixer._sdp_dim.size == 1 for block in blocks)

    def _decode_plan(self, cache: KeyValueCache):
        """Description of the decoder for the native generation step, None if some part of it has to run layer by layer.  It
        holds weight addresses, so every new request (the pass over its prompt) has the decoder described afresh."""
        if cache.length == 0:
            self._plan = None
            return None
        described = self._plan
        if described is None:
            from fast_llm_b200.engine.inference.decode import DecodePlan

            described = self._plan = (DecodePlan.build(self._model),)
        return described[0]

    @torch.no_grad()
    def forward_rows(self, tokens: torch.Tensor, cache: KeyValueCache, output_hidden_states=None):
        """`tokens` [rows, n]: the next n positions of every row of `cache` (the whole left-padded prompt when the cache is
        empty).  Returns logits [rows * n, vocab] (and the hidden states asked for) and extends the cache."""
        from fast_llm_b200.layers.kwargs import LanguageModelKwargs

        rows, new = tokens.shape
        assert rows == cache.rows
        if not output_hidden_states and (plan := self._decode_plan(cache)) is not None and plan.takes(rows, new, cache):
            return plan.step(tokens, cache, self._distributed.device), {}
        held = cache.length
        cu_q, cu_k, positions, documents = [0], [0], [], []
        for pad in cache.pads:
            pad_queries = pad if held == 0 else 0  # the padding is only ever seen by itself, in the first pass
            if pad:
                cu_q.append(cu_q[-1] + pad_queries)
                cu_k.append(cu_k[-1] + pad)
                positions.append(torch.arange(pad_queries))
                documents += [len(cu_q) - 2] * pad_queries
            queries, seen = new - pad_queries, max(held - pad, 0)  # `seen`: real positions of this row in the cache
            cu_q.append(cu_q[-1] + queries)
            cu_k.append(cu_k[-1] + seen + queries)
            positions.append(torch.arange(seen, seen + queries))
            documents += [len(cu_q) - 2] * queries
        lengths_q = [b - a for a, b in zip(cu_q, cu_q[1:])]
        lengths_k = [b - a for a, b in zip(cu_k, cu_k[1:])]
        device = self._distributed.device
        kwargs = {
            LanguageModelKwargs.token_ids: tokens.reshape(-1).to(device),
            LanguageModelKwargs.position_ids: torch.cat(positions).to(device=device, dtype=torch.int32),
            LanguageModelKwargs.document_index: torch.tensor(documents, dtype=torch.int32, device=device),
            LanguageModelKwargs.cu_seqlens_q: torch.tensor(cu_q, dtype=torch.int32, device=device),
            LanguageModelKwargs.cu_seqlens_k: torch.tensor(cu_k, dtype=torch.int32, device=device),
            LanguageModelKwargs.max_seqlen_q: max(lengths_q), LanguageModelKwargs.max_seqlen_k: max(lengths_k),
            LanguageModelKwargs.num_tokens: rows * new, LanguageModelKwargs.micro_sequence_index: 0,
            LanguageModelKwargs.sequence_k_offset: rows * (held + new), "max_position": held + new,
            LanguageModelKwargs.key_value_rows: rows, LanguageModelKwargs.presents: [], "return_logits": True,
        }
        if held:
            kwargs[LanguageModelKwargs.past_key_values] = list(cache.layers)
        if output_hidden_states:
            kwargs["output_hidden_states"] = set(output_hidden_states)
            kwargs["hidden_states"] = {}
        for layer in self._model.base_model.get_layers():
            layer.preprocess(kwargs)
        self.forward_kwargs(kwargs[LanguageModelKwargs.token_ids], kwargs)
        cache.layers = [kv.detach() for kv in kwargs[LanguageModelKwargs.presents]]
        cache.length = held + new
        return kwargs["logits"], kwargs.get("hidden_states", {})
