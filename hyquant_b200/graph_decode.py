"""One generated token's decode attention for every layer as ONE CUDA-graph replay.

The reference appends and attends layer by layer from Python, with the cache lengths as host integers
(``src/ops/d_stage_kv_cache.py:195-303``); here the lengths travel with the step's inputs: the caller fills one pinned
host message (every layer's new q / k / v rows), :class:`DecodeStepGraph` adds every layer's ``(n_quant, n_staging)``,
and the replayed graph is copy in -> one fused append + attention launch per layer, side by side -> copy out.  The decode kernels
read the lengths from the message (``hq_decode_args.lengths``), so the same graph serves every step; only the step on
which a staging buffer fills (one in 128) runs eagerly, because it quantises 128 tokens first, and so does the first.

Every layer's rows have to be known before the step.  The layer-by-layer loop of one decoder, where the query of a layer
is made from the output of the one before, calls :meth:`DStageLayerCache.decode_step` per layer instead.
"""

from __future__ import annotations

import ctypes as C
from typing import List

import torch

from . import _lib
from ._lib import HyQuantError


class DecodeStepGraph:
    def __init__(self, layers: List, batch: int, h_q: int, h_kv: int, device=None):
        if not layers or any(l.phase != "decode" for l in layers):
            raise HyQuantError("DecodeStepGraph needs frozen layer caches")
        self.layers, self.B, self.H_Q, self.H_KV = layers, batch, h_q, h_kv
        self.R = h_q // h_kv
        dev = layers[0].k_window.device if device is None else device
        n, D = len(layers), 128
        rows = batch * (h_q + 2 * h_kv)
        self._row_bytes = rows * D * 2
        msg = n * self._row_bytes + n * 8                       # q | k | v rows of every layer, then (n_quant, n_staging) per layer
        self.host_in = torch.zeros(msg, dtype=torch.uint8).pin_memory()
        self.dev_in = torch.zeros(msg, dtype=torch.uint8, device=dev)
        self.host_out = torch.empty(n, batch, h_q, 1, D, dtype=torch.bfloat16).pin_memory()
        self.dev_out = torch.empty(n, batch, h_q, 1, D, dtype=torch.bfloat16, device=dev)

        def views(buf):
            x = buf[:n * self._row_bytes].view(torch.bfloat16).view(n, rows, D)
            q = [x[i, :batch * h_q].view(batch, h_q, 1, D) for i in range(n)]
            k = [x[i, batch * h_q:batch * (h_q + h_kv)].view(batch, h_kv, 1, D) for i in range(n)]
            v = [x[i, batch * (h_q + h_kv):].view(batch, h_kv, 1, D) for i in range(n)]
            return q, k, v, buf[n * self._row_bytes:].view(torch.int32).view(n, 2)

        self.host_q, self.host_k, self.host_v, self._host_len = views(self.host_in)     # the caller fills host_q/k/v
        self._host_len_np = self._host_len.numpy()        # same memory; element-wise tensor writes would cost microseconds each
        self._q, self._k, self._v, self._len = views(self.dev_in)
        for i, layer in enumerate(layers):
            layer.bind_lengths(self._len[i])
        self._graph = None
        self._ws, self._streams = [], []         # one split-K workspace per branch of the graph, and the branches' streams
        self._used_on = {_lib.stream_ptr(self.dev_in.device)}    # streams the device buffers are safe to be freed behind
        self._warm = False

    BRANCHES = 16

    def _plan_launches(self):
        """(splits of a head, branches of the graph; 0 splits = as a launch that has the chip for itself).

        The launches share the chip, so they run as half-size blocks, two to an SM (HQ_DECODE_SHARED_CHIP).  Splits: as many
        as give sixteen launches in flight about 1.75 blocks per place (some wait and take over where others end), or, with
        few layers, one block per place; and no more than leave a warp four units (32 quantised or 8 BF16 tokens) to
        work on.  Measured on 8 kv-heads, the replay alone: 32 layers of an 8K prefix 126 us with 4 splits (16 branches of
        full-size blocks 143 to 165), 16 layers of 16K 111 with 4 (115), 32 layers of 1K 75 with 2 to 4 (82), 8 layers of
        2K 43 with 2 to 4 (48).  A whole step() of 32 layers of 8K: 148, with one launch after the other 346."""
        branches = min(self.BRANCHES, len(self.layers))
        if branches == 1:
            return 0, 1
        sms = torch.cuda.get_device_properties(self.dev_in.device).multi_processor_count
        heads, layer = self.B * self.H_KV, self.layers[0]
        units = layer._n_quant // 32 + (layer.k_topk.shape[1] + layer.k_window.shape[1] + layer._staging_ptr) // 8
        wanted = max(round(3.5 * sms / (self.BRANCHES * heads)), 2 * sms // (len(self.layers) * heads))
        return max(1, min(18, wanted, units // 32)), branches

    def _eager(self):
        self.dev_in.copy_(self.host_in, non_blocking=True)
        for i, layer in enumerate(self.layers):
            layer.decode_step(self._q[i], self._k[i], self._v[i], self.R, out=self.dev_out[i])
        self.host_out.copy_(self.dev_out, non_blocking=True)

    def _capture(self):
        # Every layer's rows are in the message, so the layers do not wait for one another: their launches are captured on
        # sixteen branches that fork behind the input copy and join before the output copy, each branch with a split-K
        # workspace of its own (a branch's launches follow one another).  A layer is then cut into fewer, longer
        # blocks, because the other layers fill the chip.
        splits, branches = self._plan_launches()
        g = torch.cuda.CUDAGraph()
        dev = self.dev_in.device
        if not self._ws:
            nbytes = C.c_int64(0)
            _lib.check(_lib.lib().hq_decode_workspace_bytes(self.B * self.H_KV, self.R, C.byref(nbytes)), "hq_decode_workspace_bytes")
            self._ws = [torch.zeros(int(nbytes.value), dtype=torch.uint8, device=dev) for _ in range(branches)]
            self._streams = [torch.cuda.Stream(dev) for _ in range(branches - 1)]
            self._used_on = set()
        with torch.cuda.graph(g):
            main = torch.cuda.current_stream(dev)
            self.dev_in.copy_(self.host_in, non_blocking=True)
            streams = [main] + self._streams
            for s in self._streams:
                s.wait_stream(main)
            for i, layer in enumerate(self.layers):
                with torch.cuda.stream(streams[i % branches]):
                    layer.capture_decode_step(self._q[i], self._k[i], self._v[i], self.R, self.dev_out[i], overlap=False,
                                              num_splits=splits, workspace=self._ws[i % branches])
            for s in self._streams:
                main.wait_stream(s)
            self.host_out.copy_(self.dev_out, non_blocking=True)
        self._graph = g
        self._ptrs = [l._kq.data_ptr() for l in self.layers]

    def _follow_stream(self):
        """A replay may run on another stream than the one the buffers were allocated on, and it need not be over when
        :meth:`close` or the end of this object gives them back: the allocator has to know of that stream."""
        stream = _lib.stream_ptr(self.dev_in.device)
        if stream not in self._used_on:
            current = torch.cuda.current_stream(self.dev_in.device)
            for t in (self.dev_in, self.dev_out, *self._ws):
                t.record_stream(current)
            self._used_on.add(stream)

    def step(self, synchronize: bool = True) -> torch.Tensor:
        """Run one token: ``host_q / host_k / host_v`` hold the new rows of every layer; returns ``host_out``
        ([layers, B, H_Q, 1, D], valid after the stream has been synchronised)."""
        from .d_stage_kv_cache import GROUP_SIZE
        flush = False
        lens = []
        for layer in self.layers:
            nq, ns = layer._n_quant, layer._staging_ptr
            if ns >= GROUP_SIZE - 1:           # that layer appends, quantises its 128 staged tokens, then attends
                nq, ns, flush = nq + GROUP_SIZE, 0, True
            lens.append((nq, ns))
        self._host_len_np[:] = lens
        if flush or not self._warm:
            self._eager()
            self._warm = True
            if flush and self._graph is not None and self._ptrs != [l._kq.data_ptr() for l in self.layers]:
                self._graph = None             # a prefix buffer was re-allocated to grow: capture again
        else:
            if self._graph is None:
                self._capture()
            self._follow_stream()
            self._graph.replay()
            for layer in self.layers:
                layer.count_replayed_step()
        if synchronize:
            torch.cuda.current_stream().synchronize()
        return self.host_out

    def close(self):
        for layer in self.layers:
            layer.bind_lengths(None)
        self._graph = None
        self._ws, self._streams = [], []
