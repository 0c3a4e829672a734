"""The step function shared by the layer-list decoders of the generation path (Kelutar, Golavik, Gubulorn, Tokatar,
Manapel, Buvesun): one `step()` runs a PACKED batch (llark_b200.state_cache) -- requests that start, go on by a portion of their prompt or decode one token are
the same kernels with other numbers -- and returns fp32 logits for the rows that are asked for. A model's engine
subclasses this and says how tokens become the residual stream (`_embed`), what its layers do to it (`_run_layers`) and
how wanted rows become logits (`_logits`); slot handling, the step descriptor, validation and the order of things are
here. The engine is host-side orchestration only, like LlamaEngine: every FLOP is a C-ABI call."""
import numpy as np
import torch

F32 = torch.float32


def _flat(tokens):
    """The token ids of all requests in one integer array."""
    try:
        parts = [np.array(t, dtype=np.int64) for t in tokens]
        if all(p.ndim == 1 for p in parts):
            return np.concatenate(parts)
    except (TypeError, ValueError, OverflowError, RuntimeError):
        pass  # ids that numpy does not take as they are
    return np.array([int(t) for ts in tokens for t in ts], dtype=object)


class LayerListEngine:
    max_positions = None  # most tokens a request may hold (None: no bound)

    def _init_device(self, device, dtype):
        dev = torch.device(device)
        if dev.type != "cuda":
            raise RuntimeError("llark_b200 has no CPU path: the engine needs a CUDA device (B200)")
        if dtype not in (torch.bfloat16, torch.float32):
            raise TypeError("dtype must be torch.bfloat16 or torch.float32")
        self.device, self.act = dev, dtype
        return dev

    # hooks ------------------------------------------------------------------------------------------------------
    def new_cache(self, n_slots=4):
        raise NotImplementedError

    def _embed(self, ids, st):
        raise NotImplementedError

    def _run_layers(self, cache, x, st, residuals):
        """x fp32 [n_tok, width] through every layer; appends the stream after each layer run to `residuals` if given."""
        raise NotImplementedError

    def _logits(self, x, rows):
        raise NotImplementedError

    # one step ---------------------------------------------------------------------------------------------------
    @torch.no_grad()
    def step(self, cache, slots, tokens, want=None, return_residuals=False):
        """slots: the requests of this step; tokens[b]: the next token ids of request slots[b] (they continue at the
        position where the request stopped); want[b]: indices into tokens[b] whose logits are asked for (None: the last
        one of each). Returns fp32 logits [n_wanted, vocab] in the order of the requests and of `want` (None when nothing
        is wanted). The caches advance by the step's tokens."""
        lens = [len(t) for t in tokens]
        cache.check(slots)
        if not lens or min(lens) <= 0:
            raise ValueError("a step needs at least one token for every request in it")
        if self.max_positions is not None:
            for s, n in zip(slots, lens):
                if cache.length[s] + n > self.max_positions:
                    raise ValueError("a request grows past max_positions")
        cache.reserve_positions(max(cache.length[s] + n for s, n in zip(slots, lens)))  # per-position stores grow first
        flat = _flat(tokens)
        if flat.min() < 0 or flat.max() >= self.cfg.vocab:
            raise ValueError("token id outside the vocabulary")
        if want is None:
            want = [[n - 1] for n in lens]
        rows, first = [], [0]
        for n in lens:
            first.append(first[-1] + n)
        for b, w in enumerate(want):
            for k in w:
                if k < 0 or k >= lens[b]:  # IndexError for a request that is not in the step
                    raise ValueError("a wanted place lies outside the request's tokens")
                rows.append(first[b] + int(k))
        st = cache.layout(slots, lens, extra=(flat, rows))
        ids, idx = st.extra
        x = self._embed(ids, st)
        residuals = [] if return_residuals else None
        x = self._run_layers(cache, x, st, residuals)
        cache.advance(slots, lens)
        logits = None
        if rows:
            logits = self._logits(x, idx)
        if return_residuals:
            return logits, residuals
        return logits
