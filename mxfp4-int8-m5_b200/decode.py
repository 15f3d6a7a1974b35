"""Batch-1 decode (token generation) with W4A8 GEMVs that read the packed 4-bit weights directly: the torch counterpart of
the reference's DecodeQwen3 / DecodeOlmoe (e2e/decode.py:29-165) over libscmx.  The linears compute the same function as
the prefill path (same INT8 activations, exact integer totals, same epilogues).

Attention at L = 1 is the library's own decode-attention kernel (attention="kernel"), which reads the sequence length on
the device, or torch's (attention="torch").  With the kernel, a whole step - embedding, every layer, output head, argmax,
position counter - is captured in one CUDA graph (`generate`) and replayed per token; the reference reaches the same end
by mx.compile'ing the halves of a step (e2e/decode.py:31-33).

fuse_prologue selects where the per-token INT8 of a GEMV input is computed in the reference (inside the GEMV or in a row
kernel); here both forms run the row kernel followed by the GEMV and give the same values, so the argument only keeps the
signature.

persistent=True (DecodeQwen3) runs all layers of a step as ONE cooperative kernel (scmx_decode_step): rows travel between
the phases of a layer as packets instead of across kernel boundaries, each CTA re-quantizes the activations it needs in
shared memory, and weights stream ahead of the phases.  Same bits as the chain of kernels; used where its limits
hold (head size 128, widths multiples of 1024 up to 6144, shares of rows that fit the multiprocessors) and attention="kernel".

DecodeHybrid is the same for hybrid decoders (fused_hybrid.FusedHybrid): GEMVs on bfloat16 or float32 weights with the mixers'
one-token kernels between them, float32 activations."""
import ctypes

import numpy as np
import torch

from . import _lib
from . import sc_decode as G
from . import sc_kernels as S
from . import hybrid_mixers as MX
from . import sc_mixers as X
from . import sc_moe as M_


class _Decoder:
    _mk = None                                                # persistent-kernel state, built per cache

    def __init__(self, fused, head, attention):
        self.f, self.model, self.args = fused, fused.model, fused.args
        self.head = G.head_product(fused.model if head == "model" else head)
        a = self.args
        hq, hk, d = a.num_attention_heads, a.num_key_value_heads, a.head_dim
        if attention == "kernel" and not S.DecodeAttention.supports(hq, hk, d):
            attention = "torch"
        self.attention = attention
        self.attn = S.DecodeAttention(hq, hk, d, fused.inv_freq.device) if attention == "kernel" else None
        self._graph = None

    @property
    def replayable(self):
        """Whether a step reads its position on the device, so that one captured graph serves every position."""
        return self.attn is not None

    def _attend(self, at, c, q, k, v, pos_dev):
        if self.attn is not None:
            return self.attn(q, c, at.scale, n_pos=None if pos_dev is not None else c.offset + 1, pos_dev=pos_dev)
        assert pos_dev is None, "a device-side position needs attention='kernel'"
        return self.f.sdpa(q, k, v, at.scale, False)

    @torch.no_grad()
    def step(self, tok, cache):
        """tok int [1, 1] -> logits [1, 1, V]; appends one position to the cache."""
        logits = self._step(tok, cache, None)
        for c in cache:
            c.offset += 1
        return logits

    @torch.no_grad()
    def generate(self, tok, cache, n):
        """Greedy decoding of n tokens after `tok` (int [1, 1]) from one captured CUDA graph replayed n times.
        Returns int64 [n]; the cache advances by n positions."""
        assert self.replayable, "graph decoding needs attention='kernel'"
        dev = tok.device
        if self._graph is None or self._graph[0] is not cache:
            offsets = [c.offset for c in cache]
            # the warm-up run below writes the cache row at `pos`: point it at the row the first real step overwrites
            tok_buf = tok.reshape(1, 1).to(torch.long).clone()
            pos = torch.full((1,), offsets[0], dtype=torch.int32, device=dev)
            count = torch.zeros(1, dtype=torch.int32, device=dev)
            chosen = torch.empty(cache[0].capacity, dtype=torch.long, device=dev)
            for c in cache:
                c.offset = 0                                   # rows and rotary positions come from `pos` on the device
            s = torch.cuda.Stream(device=dev)
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                kept = [(t, t.clone()) for c in cache for t in c.carried()]
                logits = self._step(tok_buf, cache, pos)       # warm-up outside the capture (lazy initialisations)
                self._select(logits, tok_buf, pos, count, chosen)
                for t, old in kept:                            # recurrent states must not see the warm-up token
                    t.copy_(old)
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    logits = self._step(tok_buf, cache, pos)
                    self._select(logits, tok_buf, pos, count, chosen)
            torch.cuda.current_stream().wait_stream(s)
            for c, o in zip(cache, offsets):
                c.offset = o
            self._graph = (cache, g, tok_buf, pos, count, chosen, logits, self._mk)
        # the layer table, scratch and status word that the graph names live as long as it does, whatever cache was stepped on since
        _, g, tok_buf, pos, count, chosen, _, self._mk = self._graph
        start = cache[0].offset
        assert start + n <= cache[0].capacity, "KV cache capacity exceeded"
        tok_buf.copy_(tok.reshape(1, 1))
        pos.fill_(start)
        count.zero_()
        for _ in range(n):
            g.replay()
        out = chosen[:n].clone()
        for c in cache:
            c.offset = start + n
        return out


    _call = staticmethod(_lib.call)      # the library that the decoder's kernels are in

    def _select(self, logits, tok, pos, count, chosen):
        """The next token (greedy) as the step's input and in the list of chosen ones, and the step's counters, in one kernel."""
        row = logits[:, -1].reshape(-1)
        if row.dtype not in (torch.bfloat16, torch.float32):      # a head of its own
            tok.copy_(row.argmax(-1, keepdim=True).view_as(tok))
            chosen.index_copy_(0, count.long(), tok.view(1))
            count.add_(1)
            pos.add_(1)
            return
        self._call("scmx_select_token", _lib.ptr(row), int(row.dtype == torch.float32), row.numel(), _lib.ptr(tok), _lib.ptr(pos), _lib.ptr(count),
                   _lib.ptr(chosen), chosen.numel(), _lib.stream())


class DecodeQwen3(_Decoder):
    """Built from a FusedQwen3 with epilogue="gemm" (gate/up rows interleaved for the SwiGLU epilogue)."""

    def __init__(self, fused, head="model", compiled=True, fuse_prologue=None, act_tile=None, attention="kernel",
                 persistent=True):
        assert fused.epilogue == "gemm"
        super().__init__(fused, head, attention)
        a = self.args
        fits = lambda n: n % 1024 == 0 and n <= 6144  # noqa: E731
        self.persistent = bool(persistent and self.attn is not None and a.head_dim == 128 and fits(a.hidden_size)
                               and fits(a.intermediate_size) and fits(a.num_attention_heads * a.head_dim)
                               and a.num_attention_heads <= 32 and fused.fmt == type(fused.fmt)()
                               and (not torch.cuda.is_available() or self._shares_fit(a, self.attn.nsplit, _lib.sm_count())))

    @staticmethod
    def _shares_fit(a, nsplit, n_sm):
        """Whether the one-kernel step takes n_sm multiprocessors, as a partition of the device may have fewer: each has rows of every product, at most
        384 of one, and there is one for every query head and every split of a key/value head (scmx_decode_step)."""
        hq, hk, d = a.num_attention_heads, a.num_key_value_heads, a.head_dim
        groups = [n // 4 for n in ((hq + 2 * hk) * d, 2 * a.intermediate_size, a.hidden_size)]
        return max(hk * nsplit, hq) <= n_sm <= min(groups) and 4 * -(-max(groups) // n_sm) <= 384

    def _persistent_state(self, cache):
        """Layer table (device pointers of the packed weights, norms and this cache's tensors) and scratch buffers."""
        if self._mk is not None and self._mk["cache"] is cache:
            return self._mk
        f, a = self.f, self.args
        dev = f.inv_freq.device
        table = (_lib.ScmxDecodeLayer * len(f.layers))()
        for i, (layer, ws) in enumerate(f.layers):
            t, at, c = table[i], layer.self_attn, cache[i]
            for j, g in enumerate(("qkv", "o", "gu", "down")):
                t.codes[j], t.bcodes[j], t.wscale[j] = ws[g].codes.data_ptr(), ws[g].bcodes.data_ptr(), ws[g].wscale.data_ptr()
            t.ln_in, t.ln_post = layer.input_layernorm.weight.data_ptr(), layer.post_attention_layernorm.weight.data_ptr()
            t.q_norm, t.k_norm = at.q_norm.weight.data_ptr(), at.k_norm.weight.data_ptr()
            t.k_cache, t.v_cache = c.k.data_ptr(), c.v.data_ptr()
        raw = np.frombuffer(ctypes.string_at(ctypes.addressof(table), ctypes.sizeof(table)), dtype=np.uint8).copy()
        size = _lib.lib().scmx_decode_step_scratch(a.hidden_size, a.intermediate_size, a.num_attention_heads, a.num_key_value_heads, a.head_dim, self.attn.nsplit)
        self._mk = dict(cache=cache, table=torch.from_numpy(raw).to(dev), scratch=torch.zeros(size, dtype=torch.uint8, device=dev),
                        status=torch.zeros(1, dtype=torch.int32, device=dev),
                        pos=torch.zeros(1, dtype=torch.int32, device=dev))
        return self._mk

    def check_status(self):
        """Raises if a wait of the persistent kernel timed out (synchronizes)."""
        if self._mk is not None:
            st = int(self._mk["status"].item())
            if st:
                raise _lib.ScmxError(f"persistent decode kernel: {_lib.describe_status(st)}")

    def _step_persistent(self, tok, cache, pos_dev):
        f, a = self.f, self.args
        mk = self._persistent_state(cache)
        if pos_dev is None:
            pos_dev = mk["pos"]
            pos_dev.fill_(cache[0].offset)
        hq, hk, d = a.num_attention_heads, a.num_key_value_heads, a.head_dim
        h = self.model.model.embed_tokens(tok)[0].clone()     # [1, D]; the kernel updates it in place
        _lib.call("scmx_decode_step", _lib.ptr(mk["table"]), len(f.layers), a.hidden_size, a.intermediate_size, hq, hk, d,
                  float(f.eps), float(f.layers[0][0].self_attn.scale), _lib.ptr(f.inv_freq), _lib.ptr(f.rope_cs),
                  f.rope_cs.shape[0], cache[0].k.shape[1], _lib.ptr(pos_dev), _lib.ptr(h), _lib.ptr(mk["scratch"]), self.attn.nsplit,
                  _lib.ptr(mk["status"]), _lib.stream())
        xn = S.rmsnorm_quant_n(h, self.model.model.norm.weight, f.eps, 1)[2]
        return self.head(xn[None])

    def _step(self, tok, cache, pos_dev):
        f, a = self.f, self.args
        S.set_format(f.fmt)
        if self.persistent:
            return self._step_persistent(tok, cache, pos_dev)
        hq, hk, d, eps = a.num_attention_heads, a.num_key_value_heads, a.head_dim, f.eps
        h = self.model.model.embed_tokens(tok)[0]             # [1, D]
        for i, (layer, ws) in enumerate(f.layers):
            at, c = layer.self_attn, cache[i]
            w = ws["qkv"]
            y = G.gemv(h, w.codes, w.bcodes, None, w.wscale, w.N, 1, pro=2, nw=layer.input_layernorm.weight, eps=eps)
            q, k, v = S.qkv_headnorm_y(y[None], at.q_norm.weight, at.k_norm.weight, eps, 1, hq, hk, d,
                                       rope=(f.inv_freq, c.offset, f.rope_cs), cache=c, pos_dev=pos_dev)
            o = self._attend(at, c, q, k, v, pos_dev)
            wo, wg, wd = ws["o"], ws["gu"], ws["down"]
            h = G.gemv(o, wo.codes, wo.bcodes, None, wo.wscale, wo.N, 2, res=h, pro=1)[None]
            act = G.gemv(h, wg.codes, wg.bcodes, None, wg.wscale, wg.N, 3, pro=2, nw=layer.post_attention_layernorm.weight,
                         eps=eps)
            h = G.gemv(act[None], wd.codes, wd.bcodes, None, wd.wscale, wd.N, 2, res=h, pro=1)[None]
        xn = S.rmsnorm_quant_n(h, self.model.model.norm.weight, eps, 1)[2]
        return self.head(xn[None])


class DecodeOlmoe(_Decoder):
    """Built from a FusedOlmoe: the expert GEMVs gather the top-k experts' rows themselves."""

    def __init__(self, fused, head="model", compiled=True, fuse_prologue=False, o_tile=None, attention="kernel"):
        super().__init__(fused, head, attention)
        assert not self.args.norm_topk_prob
        self.pos = torch.arange(self.args.num_experts_per_tok, dtype=torch.int32, device=fused.inv_freq.device)

    def _step(self, tok, cache, pos_dev):
        f, a = self.f, self.args
        H, d, D, eps = a.num_attention_heads, a.head_dim, a.hidden_size, f.eps
        F2, k = 2 * a.intermediate_size, a.num_experts_per_tok
        h = self.model.model.embed_tokens(tok)[0]
        row = out = None
        for i, (layer, ws, ex) in enumerate(f.layers):
            at, c = layer.self_attn, cache[i]
            w, wo = ws["qkv"], ws["o"]
            if row is None:
                y = G.gemv(h, w.codes, w.bcodes, None, w.wscale, 3 * H * d, 1, pro=2, nw=layer.input_layernorm.weight, eps=eps)
            else:
                y = G.gemv(row[0], w.codes, w.bcodes, row[1], w.wscale, 3 * H * d, 1)
            q, kk, v = S.qkv_fullnorm_y(y[None], at.q_norm.weight, at.k_norm.weight, eps, 1, H, d,
                                        rope=(f.inv_freq, c.offset, f.rope_cs), cache=c, pos_dev=pos_dev)
            o = self._attend(at, c, q, kk, v, pos_dev)
            h = G.gemv(o, wo.codes, wo.bcodes, None, wo.wscale, D, 2, res=h, pro=1)[None]
            pn = layer.post_attention_layernorm.weight
            xq, xs, inds, scores = f.norm_route_token(layer, h)
            e = inds.reshape(-1)
            (cg, bg, sg), (cd, bd, sd) = ex["gu"], ex["down"]
            act = G.gemv(xq, cg, bg, xs, sg, F2, 3, eidx=e, xstride=0)            # [k, F]
            yd = G.gemv(act, cd, bd, None, sd, D, 1, eidx=e, xstride=1, pro=1)    # [k, D], per-row INT8 in the prologue
            # the sum of the experts' rows and the norm that follows: the next layer's INT8 row, or the output head's row
            last = i + 1 == len(f.layers)
            nn = self.model.model.norm.weight if last else f.layers[i + 1][0].input_layernorm.weight
            if D <= 8192:
                h, *row, out = M_.combine_norm(yd, self.pos, scores, h, nn, eps, quant=not last, normed=last)
            else:
                h = M_.moe_combine(yd, self.pos, scores, h, pn, eps, 1, quant=False)[0]
        return self.head((S.rmsnorm_quant_n(h, self.model.model.norm.weight, eps, 1)[2] if out is None else out)[None])


def _row(row, in_parts):
    """A row for its reader: as it is left, or joined."""
    return row if in_parts or not isinstance(row, X.RowParts) else row.joined()


class DecodeHybrid(_Decoder):
    """Built from a FusedHybrid.  Activations of a step are float32 vectors in buffers that live with the decoder."""
    replayable = True
    _call = staticmethod(_lib.mcall)

    def __init__(self, fused):
        self.f, self.model, self.args, self._graph = fused, fused.model, fused.args, None
        dev, a = fused.model.device, self.args
        f32 = lambda *s: torch.empty(s, dtype=torch.float32, device=dev)    # noqa: E731
        # the residual row: a product that joins it reads one buffer and writes the other
        self.x, self.y = (f32(1, a.hidden_size), f32(1, a.hidden_size)), f32(1, a.hidden_size)
        if not a.design.prenorm:     # the embedding's and every layer's result, for the depth average
            self.xs = f32(len(a.layers) + 1, 1, a.hidden_size)
        own = {}
        for ly in fused.layers:
            if ly not in own:
                own[ly] = ly.mixer.buffers(dev)
                if ly.w_up is not None:
                    own[ly]["u"] = f32(ly.w_up.N // (2 if ly.act.code == 2 else 1))
        self.bufs = [own[ly] for ly in fused.layers]

    def _mix(self, ly, b, x, c, pos_dev):
        x = _row(x, MX.reads_parts(ly.mixer))
        return ly.mixer.w_o.vec(ly.mixer.step(self.f, x, c, b, pos_dev), out=self.y.view(-1))

    def _step(self, tok, cache, pos_dev):
        f = self.f
        f.ensure_positions(cache[0].capacity)
        assert pos_dev is not None or cache[0].offset < cache[0].capacity, "KV cache capacity exceeded"
        row = (self._prenorm if self.args.design.prenorm else self._postnorm)(tok.view(-1), cache, pos_dev)
        return f.head.vec(_row(row, X.reads_parts(f.head)))[None, None]

    def _prenorm(self, tok, cache, pos_dev):
        f, (x, spare), y, mult = self.f, self.x, self.y, self.args.residual_mult
        f.embed(tok, cache, x)
        nl = len(f.layers)
        row = X.RowParts(x, None, f.layers[0].norm1 if nl else f.final_norm, mult, f.eps, None)
        for i, (ly, b, c) in enumerate(zip(f.layers, self.bufs, cache)):
            after = f.layers[i + 1].norm1 if i + 1 < nl else f.final_norm
            self._mix(ly, b, row, c, pos_dev)
            row, x, spare = X.RowParts(x, y, after if ly.w_up is None else ly.norm2, mult, f.eps, spare), spare, x
            if ly.w_up is not None:
                ly.feed_forward_vec(_row(row, ly.feed_reads_parts()), b["u"], y.view(-1))
                row, x, spare = X.RowParts(x, y, after, mult, f.eps, spare), spare, x
        return row

    def _postnorm(self, tok, cache, pos_dev):
        f, y, nl = self.f, self.y, len(self.f.layers)
        f.embed(tok, cache, self.xs[0])
        x, row, turn = self.xs[0], self.xs[0].view(-1), 0
        if nl == 0:
            return X.norm_rows(x, f.final_norm, f.eps, torch.float32).view(-1)
        for i, (ly, b, c) in enumerate(zip(f.layers, self.bufs, cache)):
            self._mix(ly, b, row, c, pos_dev)
            last = i + 1 == nl
            norm = ly.norm1
            if ly.w_up is not None:
                row, x, turn = X.RowParts(x, y, norm, 1.0, f.eps, self.x[turn], ()), self.x[turn], 1 - turn
                ly.feed_forward_vec(_row(row, ly.feed_reads_parts()), b["u"], y.view(-1))
                norm = ly.norm2
            row = X.RowParts(x, y, norm, 1.0, f.eps, self.x[turn], (self.xs, ly.dwa, not last), f.final_norm if last else None)
            x, turn = self.x[turn], 1 - turn
        return row
