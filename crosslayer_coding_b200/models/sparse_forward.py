"""Sparse forward pass on sm_100a for inference and evaluation, for every sparse activation function.

The reference computes ``model(inputs)`` densely: per layer an encoder GEMM, the activation on the dense
``[B, F]`` tensor and one dense decoder GEMM per (source, target) pair over activations that are >99.9 % zeros
(clt/models/clt.py:285-300, clt/models/decoder.py:289-295).  Here the activation is a *selection* that emits a
``(token, feature, value)`` list and the decoder is a gather over the listed rows:

    encoder_gemm (tcgen05)  ->  selection  ->  CSR by token  ->  sparse decode (+ per-layer squared error)

Selections:
  * ``batchtopk``  global top ``k*B`` of the per-feature batch z-scores (same kernels as the training step),
  * ``topk``       every token's top ``k`` of the same z-scores (exact per-token radix selection),
  * ``jumprelu``   ``x >= exp(log_threshold[l, f])``   (the form a converted BatchTopK model is deployed in),
  * ``relu``       ``x > 0`` (only useful while the activations are sparse; dense layers overflow the list and
                   the call reports it, see ``check_status``).
Skip connections and tensor-parallel groups are not covered here; ``supports`` says so and
callers use ``CrossLayerTranscoder.forward`` for those.
"""
from __future__ import annotations

import threading
from typing import Dict, Optional

import torch

from ..ops import ext as ext_mod

_MIN_POSITIVE_BF16 = 9.183549615799121e-41  # 2**-133, the smallest positive bf16 (subnormal)


def supports(model) -> Optional[str]:
    """``None`` when ``SparseForward`` covers the model's configuration, else the reason it does not."""
    cfg = model.config
    if cfg.activation_fn not in ("batchtopk", "topk", "jumprelu", "relu"):
        return f"activation_fn={cfg.activation_fn!r}"
    if cfg.activation_fn in ("batchtopk", "topk") and cfg.topk_mode != "global":
        return "topk_mode='per_layer'"
    if cfg.skip_connection:
        return "skip_connection"
    if model.world_size > 1:
        return "tensor-parallel model"
    if model.dtype != torch.bfloat16:
        return f"model dtype {model.dtype} (needs bf16 weights)"
    if cfg.d_model % 8 != 0 or cfg.d_model > 2048 or cfg.num_layers > 32 or model.local_features % 8 != 0:
        return "shape limits (d_model % 8, d_model <= 2048, layers <= 32, features % 8)"
    if not model.enc_weight.is_cuda:
        return "model is not on a CUDA device"
    return None


class SparseForward:
    def __init__(self, model, batch_tokens: int, max_active_per_token: int = 2048, expected_active_per_token: Optional[int] = None):
        """``max_active_per_token``: room of the entry list of a threshold selection (a batch that needs more is reported, see
        ``check_status``).  ``expected_active_per_token``: about how many entries a token has under such a selection; only the speed of the
        decode depends on it (short lists take two warps per token instead of four: 4096 tokens of 12 x 768 without an entry 92 us instead
        of 114).  Left out, lists count as long unless the room says that they are not."""
        reason = supports(model)
        if reason is not None:
            raise ValueError(f"SparseForward does not cover this model: {reason}")
        self.model = model
        self.ext = ext_mod.load()
        cfg = model.config
        self.L, self.d, self.B = cfg.num_layers, cfg.d_model, int(batch_tokens)
        self.Fl = model.local_features
        self.fn = cfg.activation_fn
        self.tying = {"none": 0, "per_source": 1, "per_target": 2}[cfg.decoder_tying]
        dev = self.dev = model.enc_weight.device
        L, B, d, Fl = self.L, self.B, self.d, self.Fl
        i32, f32 = torch.int32, torch.float32
        if self.fn == "batchtopk":
            self.k_total = min(int(cfg.batchtopk_k) * B, B * L * Fl)
            cap = max(self.k_total, 8)
        elif self.fn == "topk":
            from .activations import resolve_token_k

            self.k_token = resolve_token_k(float(cfg.topk_k), L * Fl)
            self.k_total = self.k_token * B
            cap = max(self.k_total, 8)
        else:
            cap = int(min(B * L * Fl, max_active_per_token * B))
        self.cap = cap
        # entries per token, for the decode's choice of warps per token (0: not known)
        if self.fn in ("batchtopk", "topk"):
            self.expected_entries = self.k_total // max(B, 1)
        elif expected_active_per_token is not None:
            self.expected_entries = max(1, int(expected_active_per_token))
        else:
            self.expected_entries = max(1, int(max_active_per_token)) if max_active_per_token < 64 else 0
        self.preact = torch.empty(L, B, Fl, dtype=torch.bfloat16, device=dev)
        self.ctl = torch.zeros(16, dtype=torch.int64, device=dev)
        self.status = torch.zeros(4, dtype=i32, device=dev)
        self.ent_tok = torch.empty(cap, dtype=i32, device=dev)
        self.ent_col = torch.empty(cap, dtype=i32, device=dev)
        self.ent_val = torch.empty(cap, dtype=f32, device=dev)
        if self.fn in ("batchtopk", "topk"):
            self.mean = torch.empty(L, Fl, dtype=f32, device=dev)
            self.rstd = torch.empty(L, Fl, dtype=f32, device=dev)
        if self.fn == "batchtopk":
            from ..training.fused_engine import histogram_range

            self.key_lo, self.shift = histogram_range(self.k_total, B * L * Fl)
            cand_cap = int(min(B * L * Fl, max(1 << 20, 4 * self.k_total)))
            self.cand = [torch.empty(cand_cap, dtype=i32, device=dev) for _ in range(3)] + [torch.empty(cand_cap, dtype=f32, device=dev)]
            self.sel_state = torch.tensor([self.key_lo, self.shift], dtype=torch.int64, device=dev) if self.key_lo != 0 else None
            self.pool = torch.empty(4, int(min(B * L * Fl, 10 * self.k_total + (1 << 16))), dtype=i32, device=dev) if self.key_lo != 0 else None
        ncols = self.ncols = L * Fl
        # counters of the CSR build and loss sums in one buffer, cleared by one memset right in front of the build: cleared at the
        # start of the call they have left L2 by then (the encoder's weights and the pre-activations passed through it), and the
        # scan over them takes 21 us instead of 16 at 12 x 24576 features.  The loss sums come last, because only `reconstruct`
        # clears them.
        self.hist = torch.zeros(2 * 8192 + 32, dtype=i32, device=dev) if self.fn == "batchtopk" else None
        # Order: feature counters (cleared only where that view is built), token and layer counters, loss sums.
        starts = [0]
        for n in (ncols, B, L):
            starts.append((starts[-1] + n + 63) // 64 * 64)
        self._zeroed = torch.zeros(starts[-1] + 2 * L, dtype=i32, device=dev)
        self._zeroed_encode, self._zeroed_token = self._zeroed[: starts[-1]], self._zeroed[starts[1]:]
        self._feat_cnt, self.tok_cnt = self._zeroed[:ncols], self._zeroed[starts[1]: starts[1] + B]
        self.layer_cnt = self._zeroed[starts[2]: starts[2] + L]
        self.sq_err = self._zeroed[starts[-1]:].view(torch.float64)
        # see `_features`
        self._features_read = self._features_due = False
        self._lock = threading.RLock()
        self.tok_off = torch.zeros(B + 1, dtype=i32, device=dev)
        self._feat_off = torch.zeros(ncols + 1, dtype=i32, device=dev)
        self.tok_cursor = torch.zeros(B, dtype=i32, device=dev)
        self._feat_cursor = torch.zeros(ncols, dtype=i32, device=dev)
        self.tcsr_col = torch.zeros(cap, dtype=i32, device=dev)
        self.tcsr_val = torch.zeros(cap, dtype=f32, device=dev)
        self._fcsr_tok = torch.zeros(cap, dtype=i32, device=dev)
        self._fcsr_val = torch.zeros(cap, dtype=f32, device=dev)
        self.gs = torch.empty(L, B, d, dtype=torch.bfloat16, device=dev)
        if self.tying == 0:
            from .clt import pair_index

            sel = torch.zeros(L, model.num_pairs, dtype=f32, device=dev)
            for t in range(L):
                for s in range(t + 1):
                    sel[t, pair_index(s, t, L)] = 1.0
        elif self.tying == 1:
            sel = torch.tril(torch.ones(L, L, dtype=f32, device=dev))
        else:
            sel = torch.eye(L, dtype=f32, device=dev)
        self.bias_sel = sel.contiguous()
        self.bias_sum = torch.empty(L, d, dtype=f32, device=dev)
        self.theta = torch.full((L, Fl), _MIN_POSITIVE_BF16, dtype=f32, device=dev) if self.fn in ("jumprelu", "relu") else None

    # ------------------------------------------------------------------ selection
    def _theta(self) -> torch.Tensor:
        if self.fn == "jumprelu":
            # re-read on every call: the parameter may have changed.  In fp32 also for a 16-bit parameter: `exp` computes in its
            # input's type, and a threshold rounded to eight bits moves entries across it
            torch.exp(self.model.log_threshold.data.float(), out=self.theta)
        return self.theta

    @torch.no_grad()
    def encode(self, X: torch.Tensor, clear_loss: bool = False, sort_tokens: bool = True) -> None:
        """Pre-activations, selection and the token-major / feature-major CSR views of the active entries.  ``sort_tokens``: a token's
        entries ordered by (layer, feature), which the decode wants; whoever reads the feature-major view alone can do without."""
        with self._lock:
            self._select(X)
            self._build_views(clear_loss, sort_tokens)
            if not self._capturing():
                self._features_due = False

    def _build_views(self, clear_loss: bool = False, sort_tokens: bool = True) -> None:
        (self._zeroed if clear_loss else self._zeroed_encode).zero_()
        self.ext.build_csr(self.ent_tok, self.ent_col, self.ent_val, self.ctl, self.B, self.ncols, self.tok_cnt, self._feat_cnt, self.tok_off,
                           self._feat_off, self.tok_cursor, self._feat_cursor, self.tcsr_col, self.tcsr_val, self._fcsr_tok, self._fcsr_val,
                           None, 3 if sort_tokens else 2, self.Fl, self.layer_cnt)

    def _capturing(self) -> bool:
        """Whether calls on this device are being recorded into a graph (taken as true where the current device is another one)."""
        return self.dev.index not in (None, torch.cuda.current_device()) or torch.cuda.is_current_stream_capturing()

    def _features(self, name: str) -> torch.Tensor:
        """An array of the feature-major view.  It belongs to the last selection, as every other array here does, also for a caller that
        holds it over several calls.  ``reconstruct`` itself reads the token-major view alone and leaves this one out (a fifth of a
        16-token call) until somebody has asked for one of its arrays: only a caller that has asked before can hold one.  A call that is
        recorded into a graph always fills it, because nothing here learns of a replay.  The first read after calls that left it out
        builds it; which streams the list came from and the reader uses is not known here, so that read waits for the device, once
        in the life of the object."""
        with self._lock:
            self._features_read = True
            if self._features_due:
                if self._capturing():
                    self._build_views()  # recorded: every replay builds it from the list of that moment
                else:
                    torch.cuda.synchronize(self.dev)
                    self._build_views()
                    torch.cuda.synchronize(self.dev)
                    self._features_due = False
            return getattr(self, name)

    feat_off = property(lambda self: self._features("_feat_off"))
    feat_cnt = property(lambda self: self._features("_feat_cnt"))
    feat_cursor = property(lambda self: self._features("_feat_cursor"))
    fcsr_tok = property(lambda self: self._features("_fcsr_tok"))
    fcsr_val = property(lambda self: self._features("_fcsr_val"))

    def _select(self, X: torch.Tensor) -> None:
        e, m = self.ext, self.model
        assert X.dtype == torch.bfloat16 and X.shape == (self.L, self.B, self.d), (X.dtype, tuple(X.shape))
        if self.fn in ("batchtopk", "topk"):
            e.encoder_gemm_stats(X, m.enc_weight.data, m.enc_bias.data, self.preact, self.mean, self.rstd, self.status)
        else:
            e.encoder_gemm(X, m.enc_weight.data, m.enc_bias.data, self.preact, self.status, None)
        if self.fn == "batchtopk":
            self.hist.zero_()
            e.batchtopk_select(self.preact, self.mean, self.rstd, self.Fl, self.Fl, 0, self.Fl, self.k_total, self.key_lo, self.shift,
                               self.hist, self.ctl, self.ent_tok, self.ent_col, self.ent_val, self.cand[0], self.cand[1], self.cand[2],
                               self.cand[3], self.status, 1, 0, [], [], 0, 0, self.sel_state, self.pool)
        elif self.fn == "topk":
            e.token_topk_select(self.preact, self.mean, self.rstd, self.Fl, self.k_token, self.ctl, self.ent_tok, self.ent_col,
                                self.ent_val, self.status)
        else:
            e.threshold_select(self.preact, self._theta(), self.Fl, self.Fl, self.ctl, self.ent_tok, self.ent_col, self.ent_val, self.status)

    def _select_for_decode(self, X: torch.Tensor) -> None:
        """Selection and the token-major view; the feature-major one too where somebody may be holding it (see ``_features``)."""
        with self._lock:
            if self._features_read or self._capturing():
                self.encode(X, clear_loss=True)
                return
            self._select(X)
            self._zeroed_token.zero_()
            self.ext.build_token_csr(self.ent_tok, self.ent_col, self.ent_val, self.ctl, self.B, self.ncols, self.tok_cnt, self.tok_off,
                                     self.tok_cursor, self.tcsr_col, self.tcsr_val, self.layer_cnt, self.Fl)
            self._features_due = True

    # ------------------------------------------------------------------ decode
    @torch.no_grad()
    def reconstruct(self, X: torch.Tensor, Y: Optional[torch.Tensor] = None, sigma: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Reconstructions ``[L, B, d]`` (fp32).  With targets ``Y`` the per-layer sums of squared errors
        (scaled by ``sigma [L, d]`` when given) are left in ``self.sq_err``."""
        self._select_for_decode(X)
        e, m = self.ext, self.model
        yhat = torch.empty(self.L, self.B, self.d, dtype=torch.float32, device=self.dev)
        bias = m.dec_bias.data
        if bias.dtype not in (torch.bfloat16, torch.float16, torch.float32) or not bias.is_contiguous():
            bias = bias.float().contiguous()  # the types and the layout the kernel reads
        e.step_finish(None, None, bias, self.bias_sel, self.bias_sum)
        off = scale = None
        if m.feature_offset is not None:
            off = m.feature_offset.data.float().contiguous()
        if m.feature_scale is not None:
            scale = m.feature_scale.data.float().contiguous()
        sg = sigma.to(device=self.dev, dtype=torch.float32).reshape(self.L, self.d).contiguous() if sigma is not None else None
        gs, sq_err = (self.gs, self.sq_err) if Y is not None else (None, None)  # no targets: the reconstruction is the only output
        e.sparse_decode([w.data for w in m.dec_weight], self.L, self.B, self.d, self.Fl, self.tying, self.tok_off, self.tcsr_col,
                        self.tcsr_val, off, scale, None, self.bias_sum, None, Y, sg, gs, yhat, sq_err, 1, [], 0, 0, self.status,
                        expected_entries=self.expected_entries, equal_lists=self.fn == "topk")
        return yhat

    def forward_dict(self, inputs: Dict[int, torch.Tensor]) -> Dict[int, torch.Tensor]:
        """Same contract as ``CrossLayerTranscoder.forward``: ``{layer: [B, d]}`` in, reconstructions out."""
        yhat = self.reconstruct(self._stacked([inputs[l].reshape(-1, self.d) for l in range(self.L)]))
        return {l: yhat[l] for l in range(self.L)}

    def _stacked(self, rows) -> torch.Tensor:
        """``[L, B, d]`` in bf16.  Layers that already lie one after the other in one tensor (the rows of a batch that a store or a capture
        filled as ``[L, B, d]``) are taken as they are; anything else is copied."""
        first, step = rows[0], self.B * self.d
        base, shape = first.data_ptr(), (self.B, self.d)
        # consecutive addresses inside the first one's storage: the other tensors are views of the same memory
        if base % 16 == 0 and first.untyped_storage().nbytes() >= 2 * (first.storage_offset() + self.L * step) and all(
                r.dtype == torch.bfloat16 and r.shape == shape and r.is_contiguous() and r.data_ptr() == base + 2 * l * step for l, r in enumerate(rows)):
            return first.detach().as_strided((self.L, self.B, self.d), (step, self.d, 1))
        return torch.stack(rows).to(torch.bfloat16)

    # ------------------------------------------------------------------ views of the last selection
    def num_entries(self) -> int:
        return int(self.ctl[3].item())

    def l0_per_layer(self) -> torch.Tensor:
        """Mean number of active features per token and layer of the last selection."""
        return self.layer_cnt.float() / self.B

    def activations_dense(self) -> torch.Tensor:
        """Dense ``[L, B, F]`` activations of the last ``encode`` (testing)."""
        n = min(self.num_entries(), self.cap)
        out = torch.zeros(self.L, self.B, self.Fl, dtype=torch.float32, device=self.dev)
        col = self.ent_col[:n].long()
        out[col // self.Fl, self.ent_tok[:n].long(), col % self.Fl] = self.ent_val[:n]
        return out

    def check_status(self) -> None:
        code = int(self.status[0].item())
        if code != 0:
            self.status.zero_()
            names = {1: "wait timeout", 2: "entry list too small (activations too dense for the sparse path)",
                     3: "selection range", 4: "tie overflow"}
            raise RuntimeError(f"sparse forward reported '{names.get(code, code)}'")
