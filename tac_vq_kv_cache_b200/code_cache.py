"""Preallocated uint8 code store for one layer, with in-place append and attention over the codes.

Replaces the reference's decode-time ``LayerCache``
(experiments_followup_mistral/evaluate_mistral_longbench.py:29-78) and the decode
branch of its ``attention_forward`` (:112-122):

* the reference grows ``[1,H,T,S]`` code tensors with ``torch.cat`` on every token
  (:49-50, an O(T) copy per step) and additionally keeps a dense fp16 window of the
  last 4096 decoded tokens (:53-59) which its attention reads;
* here the codes live in one ``[B,H,T_max,S,G]`` buffer per side that the encode
  kernel writes at offset ``length``, and attention reads the codes themselves,
  so there is no decoded window.

``visible()`` keeps the reference's window rule ``start = max(0, length - window)``
(:62-70) and ``payload_bytes()`` its byte count (:72-73): the bytes of the stored
codes of both sides.  Rotary position embedding is not applied by the attention
kernel (keys are stored as encoded).
"""

from __future__ import annotations

import torch

from . import _lib, ops


class VQCodeCache:
    """K and V codes of one layer for a batch of sequences that advance in lockstep."""

    def __init__(
        self,
        key_tables: torch.Tensor,
        value_tables: torch.Tensor,
        *,
        batch: int,
        max_tokens: int,
        window: int | None = None,
        device: torch.device | str | None = None,
        rope_theta: float | None = None,
    ) -> None:
        """``key_tables`` / ``value_tables``: ``[H,S,G,K,d]`` masters or deployed fp16 tables.

        With ``rope_theta`` the cache holds PRE-rotary keys, like the reference's ``LayerCache``: ``attend``
        rotates every rebuilt key row at its token index (default rope of Mistral/Llama) and expects the
        query rotated at its own position.  Without it no rotary step is applied.
        """
        if key_tables.ndim != 5 or key_tables.shape != value_tables.shape:
            raise ValueError("tables must be [H,S,G,K,d] with equal K and V geometry")
        if batch <= 0 or max_tokens <= 0 or (window is not None and window <= 0):
            raise ValueError("batch, max_tokens and window must be positive")
        self.device = torch.device(device if device is not None else key_tables.device)
        self.key_tables = ops.deployed_tables(key_tables).to(self.device)
        self.value_tables = ops.deployed_tables(value_tables).to(self.device)
        heads, stages, groups, _words, sub = map(int, key_tables.shape)
        self.batch, self.heads, self.stages, self.groups, self.dim = batch, heads, stages, groups, groups * sub
        self.max_tokens = int(max_tokens)
        self.window = window
        shape = (batch, heads, self.max_tokens, stages, groups)
        self.key = torch.zeros(shape, dtype=torch.uint8, device=self.device)
        self.value = torch.zeros(shape, dtype=torch.uint8, device=self.device)
        self.length = 0
        self._range = torch.zeros(2, batch, dtype=torch.int32, device=self.device)  # [start; end) per row
        self._range_is = (0, 0)
        self._workspaces: list[torch.Tensor] = []
        self._host_key, self._host_call, self._host_buffers = None, None, None  # decode_step_host's
        self.rope = None if rope_theta is None else ops.rope_table(self.max_tokens, self.dim, float(rope_theta), self.device)

    def reset(self) -> None:
        self.length = 0

    def append(self, raw_key: torch.Tensor, raw_value: torch.Tensor, *, want_recon: bool = False):
        """Encode ``[B,H,T,D]`` rows and store their codes at positions ``length .. length+T-1``.

        Returns ``(key_recon, value_recon)`` (``None`` unless ``want_recon``), the
        quantised rows an adapter attends with during prefill.
        """
        tokens = int(raw_key.shape[2])
        if raw_key.shape != raw_value.shape or tuple(raw_key.shape[:2]) != (self.batch, self.heads) or raw_key.shape[3] != self.dim:
            raise ValueError("rows must be [B,H,T,D] matching the cache geometry")
        if self.length + tokens > self.max_tokens:
            raise ValueError("code cache is full")
        _, key_recon = ops.encode(raw_key, self.key_tables, codes=self.key, t0=self.length, want_recon=want_recon)
        _, value_recon = ops.encode(raw_value, self.value_tables, codes=self.value, t0=self.length, want_recon=want_recon)
        self.length += tokens
        return key_recon, value_recon

    def visible(self) -> tuple[int, int]:
        """Token range a decode step sees: the last ``window`` stored positions."""
        start = 0 if self.window is None else max(0, self.length - self.window)
        return start, self.length

    def payload_bytes(self) -> int:
        """Bytes of the stored K and V codes (what the reference's ledger counts)."""
        return 2 * self.batch * self.heads * self.length * self.stages * self.groups

    def attend(self, query: torch.Tensor, *, want_state: bool = False):
        """One decode step: ``query [B,Hq,D]`` fp16 (already scaled) -> fp16 ``[B,Hq,D]``.

        With ``want_state`` also returns the partial softmax state ``[B,Hq,2+D]``.
        """
        start, end = self.visible()
        if (start, end) != self._range_is:
            ops.set_ranges(self._range[0], self._range[1], start, end)
            self._range_is = (start, end)
        # work is divided as decode_step divides it; a captured call may see other ranges when it is replayed
        seen = None if self.key.is_cuda and ops._capturing(self.key.device) else end - start
        out, state = ops.attn_decode(
            query, self.key, self.value, self.key_tables, self.value_tables, self._range[0], self._range[1],
            workspace=self._scratch(int(query.shape[1])), want_state=want_state, rope=self.rope, visible=seen,
        )
        return (out, state) if want_state else out

    def decode_step(self, query: torch.Tensor, raw_key: torch.Tensor, raw_value: torch.Tensor, out: torch.Tensor | None = None):
        """Append the new token rows and attend, in one library call (``append`` + ``attend`` fused).

        ``query [B,Hq,D]`` fp16 scaled (and rotated, for a cache of pre-rotary keys), ``raw_key`` / ``raw_value``
        ``[B,H,T_new,D]`` contiguous fp16 or fp32.  The buffers, tables and window are the cache's at this call.  A cache of
        pre-rotary keys also takes what ``append`` and ``attend`` take (strided rows and queries, K and V of different
        types, no new token, strided tables) and any ``out`` that the result can be copied to: these steps are the separate calls.
        """
        batch, heads, dim = self.batch, self.heads, self.dim
        shape, q_shape, dtype = raw_key.shape, query.shape, raw_key.dtype
        if len(shape) != 4 or shape != raw_value.shape or shape[0] != batch or shape[1] != heads or shape[3] != dim:
            raise ValueError("rows must be [B,H,T,D] matching the cache geometry")
        if len(q_shape) != 3 or q_shape[0] != batch or q_shape[2] != dim or query.dtype != torch.float16:
            raise ValueError("query must be fp16 [B,Hq,D]")
        packed = raw_key.is_contiguous() and raw_value.is_contiguous() and query.is_contiguous()
        if self.rope is not None and not (packed and dtype == raw_value.dtype and shape[2] and (out is None or self._result_fits(out, query))
                                          and self.key_tables.is_contiguous() and self.value_tables.is_contiguous()):
            self.append(raw_key, raw_value)
            result = self.attend(query)
            return result if out is None else out.copy_(result)
        if dtype != raw_value.dtype or dtype not in ops._DTYPE_TAG:
            raise ValueError("rows must be of one dtype, fp16 or fp32")
        if not packed:
            raise ValueError("query and rows must be contiguous")
        ktab, vtab, rope, key, value, start, end, words, index = self._addresses()
        if not (index == query.get_device() == raw_key.get_device() == raw_value.get_device()):
            ops._require_cuda(self.key, query, raw_key, raw_value)
        if out is None:
            out = torch.empty_like(query)
        elif out.shape != q_shape or out.dtype != torch.float16 or not out.is_contiguous() or out.get_device() != index:
            raise ValueError("out must be contiguous fp16 [B,Hq,D] on the cache's device")
        tokens, q_heads = shape[2], q_shape[1]
        if self.length + tokens > self.max_tokens:
            raise ValueError("code cache is full")
        workspace = self._scratch(q_heads)
        # read by the library during the call only
        record = _lib.STEP_PLAN.pack(
            ktab, vtab, rope, key, value, start, end, workspace.data_ptr(), workspace.numel(), self.window or 0, self.max_tokens, batch, q_heads,
            heads, dim, self.groups, self.stages, words,
        )
        args = (record, query.data_ptr(), raw_key.data_ptr(), raw_value.data_ptr(), ops._DTYPE_TAG[dtype], tokens, self.length, out.data_ptr(),
                None, ops._raw_stream(index))
        if index == torch.cuda.current_device():
            status = _lib.load().tacvq_decode_step_planned(*args)
        else:
            with torch.cuda.device(index):
                status = _lib.load().tacvq_decode_step_planned(*args)
        if status:
            _lib.check("tacvq_decode_step_planned", status)
        self.length += tokens
        self._range_is = self.visible()
        return out

    @staticmethod
    def _result_fits(out: torch.Tensor, query: torch.Tensor) -> bool:
        """Whether attention may write its result to ``out`` while it reads ``query``."""
        apart = out.data_ptr() + 2 * out.numel() <= query.data_ptr() or query.data_ptr() + 2 * query.numel() <= out.data_ptr()
        return apart and out.shape == query.shape and out.dtype == torch.float16 and out.is_contiguous() and out.device == query.device

    def _addresses(self) -> tuple[int, ...]:
        """Where the K and V tables, the rotary table, the K and V codes and the range's two ends are; words a table, device.

        Asked for at every step, because a caller may put other tensors in their place; what the library would misread is refused.
        """
        ktab, vtab, rope, key, value = self.key_tables, self.value_tables, self.rope, self.key, self.value
        tokens, shape = self.max_tokens, ktab.shape
        code_shape = (self.batch, self.heads, tokens, self.stages, self.groups)
        if key.shape != code_shape or value.shape != code_shape or key.dtype != torch.uint8 or value.dtype != torch.uint8:
            raise ValueError("codes must be uint8 [B,H,T_max,S,G]")
        if len(shape) != 5 or shape != vtab.shape or ktab.dtype != torch.float16 or vtab.dtype != torch.float16:
            raise ValueError("tables must be fp16 [H,S,G,K,d]")
        heads, stages, groups, words, sub = shape
        if heads != self.heads or stages != self.stages or groups != self.groups or groups * sub != self.dim:
            raise ValueError("table and cache geometry differs")
        if not (key.is_contiguous() and value.is_contiguous() and ktab.is_contiguous() and vtab.is_contiguous()):
            raise ValueError("codes and tables must be contiguous")
        index = key.get_device()
        if not (index == value.get_device() == ktab.get_device() == vtab.get_device() >= 0) or ops._capability_major(index) != 10:
            ops._require_cuda(key, value, ktab, vtab)
        rope_at = 0
        if rope is not None:
            if rope.shape != (tokens, 2, self.dim // 2) or rope.dtype != torch.float16 or not rope.is_contiguous() or rope.get_device() != index:
                raise ValueError("rope must be contiguous fp16 [T_max, 2, D/2] on the cache's device")
            rope_at = rope.data_ptr()
        ranges = self._range.data_ptr()
        return ktab.data_ptr(), vtab.data_ptr(), rope_at, key.data_ptr(), value.data_ptr(), ranges, ranges + 4 * self.batch, words, index

    def __getstate__(self) -> dict:
        """For copies and pickles: scratch and marshalled calls stay with the cache they were made for."""
        return {**self.__dict__, "_range": self._range.clone(), "_workspaces": [], "_host_key": None, "_host_call": None, "_host_buffers": None}

    def _scratch(self, q_heads: int) -> torch.Tensor:
        """The attention workspace, large enough for ``q_heads`` query heads.

        Smaller ones are kept beside it: a captured graph goes on using the one that it was captured with.
        """
        need = ops.attn_workspace_bytes(self.batch, q_heads, self.heads, self.dim, self.groups, self.stages)
        if need == 0:
            raise ValueError("attention geometry not supported")
        if not self._workspaces or self._workspaces[-1].numel() < need:
            self._workspaces.append(torch.empty(need, dtype=torch.uint8, device=self.device))
        return self._workspaces[-1]

    def decode_step_host(self, host_rows: torch.Tensor, host_out: torch.Tensor, q_heads: int, *, tokens: int = 1,
                         synchronize: bool = True, direct: bool | str = False) -> torch.Tensor:
        """One decode step driven from HOST buffers in a single library call (``tacvq_decode_step_host``).

        ``host_rows``: pinned CPU fp16 tensor holding, back to back, the scaled query ``[B,Hq,D]``, the new K
        rows ``[B,H,tokens,D]`` and the new V rows; ``host_out``: pinned CPU fp16 ``[B,Hq,D]`` that receives the
        result.  The call enqueues the copy to the device, the encode + append + attention of
        :meth:`decode_step` and the copy back, and by default waits for them.  A decoding loop passes the same host
        buffers every step: they are checked once per pair; the cache's buffers, tables and window are those at the call.
        ``direct=True`` enqueues no copy back: the attention kernel stores the result straight into the pinned
        ``host_out`` (the rows still arrive by an enqueued copy, which was measured faster than reading them in
        place).  ``direct="rows"`` enqueues no copy at all: the kernels also read the pinned rows in place.
        """
        codes_k, codes_v, ktab, vtab = self.key, self.value, self.key_tables, self.value_tables
        # what the checked call rests on; the cache's tensors may have changed place, but not size, layout or device
        key = (host_rows.data_ptr(), host_out.data_ptr(), host_rows.nbytes, host_out.nbytes, host_rows.dtype, host_out.dtype, q_heads, tokens, direct,
               codes_k.nbytes, codes_v.nbytes, ktab.nbytes, vtab.nbytes, codes_k.get_device(), codes_v.get_device(), ktab.get_device(), vtab.get_device(),
               codes_k.is_contiguous() and codes_v.is_contiguous() and ktab.is_contiguous() and vtab.is_contiguous())
        if key != self._host_key:
            if direct not in (False, True, "rows"):
                raise ValueError('direct must be False, True or "rows"')
            self._prepare_host_call(host_rows, host_out, int(q_heads), int(tokens), direct)
            self._host_key = key
        args, call, index = self._host_call
        if self.length + tokens > self.max_tokens:
            raise ValueError("code cache is full")
        args[3:7] = ktab.data_ptr(), vtab.data_ptr(), codes_k.data_ptr(), codes_v.data_ptr()
        args[9], args[10] = self.length, self.window or 0
        args[24] = 1 if synchronize else 0
        args[25] = ops._raw_stream(index)
        if index == torch.cuda.current_device():
            status = call(*args)
        else:
            with torch.cuda.device(self.device):
                status = call(*args)
        if status:
            _lib.check("tacvq_decode_step_host", status)
        self.length += tokens
        self._range_is = self.visible()
        return host_out

    def _prepare_host_call(self, host_rows: torch.Tensor, host_out: torch.Tensor, q_heads: int, tokens: int, direct: bool | str) -> None:
        """Checks and argument marshalling of :meth:`decode_step_host`, done once per pair of host buffers."""
        if self.rope is not None:
            raise ValueError("the single-call host path has no rotary step; use append() + attend()")
        nq, nkv = self.batch * q_heads * self.dim, self.batch * self.heads * tokens * self.dim
        if host_rows.device.type != "cpu" or host_out.device.type != "cpu" or not (host_rows.is_pinned() and host_out.is_pinned()):
            raise ValueError("host_rows and host_out must be pinned CPU tensors")
        if host_rows.dtype != torch.float16 or host_out.dtype != torch.float16:
            raise ValueError("host buffers must be fp16")
        if host_rows.numel() != nq + 2 * nkv or host_out.numel() != nq or not (host_rows.is_contiguous() and host_out.is_contiguous()):
            raise ValueError("host_rows must hold q, K rows and V rows back to back; host_out must be [B,Hq,D]")
        workspace = self._scratch(q_heads)
        dev_rows = None if direct == "rows" else torch.empty(nq + 2 * nkv, dtype=torch.float16, device=self.device)
        dev_out = None if direct else torch.empty(nq, dtype=torch.float16, device=self.device)
        _, _, _, _, _, start, end, words, index = self._addresses()
        # tables, codes, length and window are filled in at every call
        args = [host_rows.data_ptr(), ops._ptr(dev_rows), ops._DTYPE_TAG[torch.float16], 0, 0, 0, 0, start, end, 0, 0, workspace.data_ptr(),
                workspace.numel(), ops._ptr(dev_out), host_out.data_ptr(), self.batch, q_heads, self.heads, self.dim,
                self.groups, self.stages, words, tokens, self.max_tokens, 1, 0]
        self._host_buffers = (dev_rows, dev_out, workspace, self._range)  # keep what the call points at alive
        self._host_call = (args, _lib.load().tacvq_decode_step_host, index)
