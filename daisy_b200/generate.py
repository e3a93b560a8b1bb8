"""Host orchestration of prefill and per-token steps over the ring cache.

Mirror of the reference ``Generator._prefill`` / ``Generator._step`` (inference/generate.py:220-248) for a
stack of attention layers: prefill fills the ring layer by layer from inside the projection kernel (the rows
``bulk_write_packed`` would write, no copy pass); each step is one launch that takes every layer's ring in place (no
per-layer chronological ``view`` copy, no separate ``write``) and advances once.
Sampling, embeddings and the MLPs are outside this path; the runner works on hidden states.
"""
from __future__ import annotations

from typing import List, Optional, Sequence

import torch

from ._lib import QKV_DEFAULT, WRITE_RING
from ._native import ext
from .attention import B200CausalSelfAttention, WindowMask
from .kv_cache import B200KVCache


class StepRunner:
    def __init__(self, layers: Sequence[B200CausalSelfAttention], window: int, cache_capacity: Optional[int] = None,
                 batch: int = 1, device="cuda", dtype=torch.bfloat16):
        assert len(layers) > 0
        self.layers = list(layers)
        self.window = int(window)
        a = self.layers[0]
        cap = int(cache_capacity if cache_capacity is not None else window)
        self.cache = B200KVCache(L=len(self.layers), B=batch, H=a.num_heads, W=cap, D=a.head_dim, device=device, dtype=dtype)

    def reset_history(self):
        self.cache.reset_history()
        for a in self.layers:
            a.reset_history()

    @torch.inference_mode()
    def _prefill(self, x: torch.Tensor) -> torch.Tensor:
        """``x [B,T,dim]`` through every layer's ``prefill`` (each layer sees the previous layer's output),
        the cache receives the rows ``Generator._prefill`` stores through ``bulk_write_packed``."""
        T, c, a = x.size(1), self.cache, self.layers[0]
        if x.is_cuda and x.size(0) == c.B and self._plain():               # the same launches, issued by one native call
            rot = [m._modules["rotary"]._buffers for m in self.layers]
            if T >= 1 and all(r["cos"].size(0) >= T for r in rot):
                r = min(T, max(c.W - 1, 0))
                x = ext().attn_stack(x, [m._parameters["qkvo_w"] for m in self.layers], [r_["cos"] for r_ in rot], [r_["sin"] for r_ in rot],
                                     a.num_heads, a.norm_eps, a.attn_scale, self.window, c.k, c.v, T - r if r > 0 else -1)
                c.set_position(T)
                return x
        for i, a in enumerate(self.layers):
            # the projection's epilogue stores the rows bulk_write_packed keeps straight into their ring slots
            x, _, _ = a.prefill_ring(x, None, self.cache, i, attn_mask=WindowMask(self.window))
        self.cache.set_position(T)
        return x

    # ------------------------------------------------------------------ all layers in one launch
    def _plain(self) -> bool:
        """Plain layers of one shape with the same constants."""
        a = self.layers[0]
        return all(type(m) is B200CausalSelfAttention and not m.receives_ve and m.num_heads == a.num_heads
                   and m.attn_scale == a.attn_scale and m.norm_eps == a.norm_eps for m in self.layers)

    def _one_launch(self, x: torch.Tensor) -> bool:
        """Whether the whole stack fits the single-launch step."""
        c = self.cache
        return x.size(0) == c.B and self._plain() and ext().token_step_supported(c.B, c.H, len(self.layers))

    def _token(self, x, t, t_dev, out=None, workspace=None):
        c, a = self.cache, self.layers[0]
        rot = [m._modules["rotary"]._buffers for m in self.layers]
        return ext().token_step(x, [m._parameters["qkvo_w"] for m in self.layers], [r["cos"] for r in rot], [r["sin"] for r in rot],
                                c.k, c.v, t, t_dev, c.t_dev, self.window, a.attn_scale, a.norm_eps, QKV_DEFAULT | WRITE_RING,
                                None, None, None, None, out, workspace)

    # ------------------------------------------------------------------ fixed-buffer step
    @torch.inference_mode()
    def capture_step(self, batch: int, dim: int) -> None:
        """Prepare ``_step_graph``: the position lives in ``cache.t_dev``, the output is a fixed buffer, nothing is allocated
        per token.  Where the stack fits the single-launch kernel that launch is the whole step; otherwise one token step
        of all layers is recorded into a CUDA graph, and ``_step_graph`` costs one copy and one graph launch per token."""
        dev = self.cache.device
        self._gx = torch.zeros(batch, 1, dim, device=dev, dtype=torch.bfloat16)
        self._graph = None
        if self._one_launch(self._gx):
            self._gy = torch.zeros_like(self._gx)
            self._gws = torch.zeros(ext().token_workspace_bytes(batch, self.cache.H), dtype=torch.uint8, device=dev)
            return
        t_saved = self.cache.t_dev.clone()
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):                              # warm-up outside the capture (lazy initialisation);
            self._graph_body(write_ring=False)                     # it must not store its dummy row into the ring
        torch.cuda.current_stream(dev).wait_stream(side)
        self.cache.t_dev.copy_(t_saved)                            # the warm-up advanced the device counter
        self._graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self._graph):
            self._gy = self._graph_body()
        self.cache.t_dev.copy_(t_saved)

    def _graph_body(self, write_ring: bool = True) -> torch.Tensor:
        x = self._gx
        for i, a in enumerate(self.layers):
            x = a.step_ring_dev(x, self.cache, i, self.window, write_ring=write_ring)
        self.cache.t_dev += 1
        return x

    @torch.inference_mode()
    def _step_graph(self, x: torch.Tensor) -> torch.Tensor:
        """``_step`` into the fixed buffer; ``x`` may lie on the host or broadcast to ``[batch, 1, dim]``.  Neither the warm-up run (made without the ring store) nor the
        capture itself (which executes nothing) has touched the ring, so a capture is safe at any position, also
        with a window larger than the ring, where the slot of the next token is the oldest row still attended."""
        if self._graph is None:
            if x.get_device() != self._gx.get_device() or x.shape != self._gx.shape:
                x = self._gx.copy_(x)
            self._token(x, 0, self.cache.t_dev, self._gy, self._gws)
        else:
            self._gx.copy_(x)
            self._graph.replay()
        self.cache.t += 1                                          # host mirror; the device counter moved in the launch
        return self._gy

    @torch.inference_mode()
    def _step(self, x: torch.Tensor) -> torch.Tensor:
        """One token ``x [B,1,dim]``: every layer reads the ring in place and stores its new row; one advance."""
        pos = self.cache.t
        if self._one_launch(x):
            torch._assert(pos < self.layers[0].rotary.cos.shape[0], "Rotary buffers too small")
            x = self._token(x, pos, None)
            self.cache.t += 1                                      # its device counter moved in the launch
            self.cache._staged = [False] * self.cache.L
            return x
        for i, a in enumerate(self.layers):
            x, _, _ = a.step_ring(x, self.cache, i, pos, None, self.window)
        self.cache.advance()
        return x
