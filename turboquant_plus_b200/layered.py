"""A stack of per-layer paged caches with a per-layer (K format, V format) table, and a decode step
that takes host buffers: copy in, quantize-on-append + attention for every layer (one CUDA graph),
copy out.  Covers asymmetric K/V formats and boundary layers kept at higher precision
(the reference's layer-aware policy: docs/papers/layer-aware-v-compression.md:25-28).
"""
from __future__ import annotations

import contextlib
import gc

from . import _native as nv
from .paged import PagedKVCache


@contextlib.contextmanager
def _capture(torch, graph):
    """torch.cuda.graph without the cyclic collector: what it frees -- another cache's graphs, events of pinned host
    buffers -- makes CUDA calls that are not allowed while a stream is capturing, and a failure inside a tensor's
    destructor ends the process."""
    enabled = gc.isenabled()
    gc.disable()
    try:
        with torch.cuda.graph(graph):
            yield
    finally:
        if enabled:
            gc.enable()


def boundary_format_table(num_layers: int, inner=("q8_0", "turbo2"), boundary=("q8_0", "q8_0"), keep: int = 2):
    """First and last ``keep`` layers use ``boundary``, the rest ``inner``."""
    return [boundary if (i < keep or i >= num_layers - keep) else inner for i in range(num_layers)]


class LayeredKVCache:
    def __init__(self, num_layers: int, head_dim: int, num_kv_heads: int, num_pages: int, page_tokens: int = 128,
                 formats=("turbo3", "turbo3"), seed: int = 42, norm_correction: bool = True,
                 rotation: str = "wht", device=None):
        if isinstance(formats[0], str):
            formats = [tuple(formats)] * num_layers
        assert len(formats) == num_layers
        self.formats = [tuple(f) for f in formats]
        # Layers of one (K format, V format) pair share the quantizers and one pool tensor: layer j of the group owns
        # pages [j * num_pages, (j + 1) * num_pages) of it.  `groups` holds, per pair, a cache object over the whole
        # tensor, through which one launch appends a token to every layer of the group.
        self.layers = [None] * num_layers
        self.groups = []
        by_format = {}
        for i, fmt in enumerate(self.formats):
            by_format.setdefault(fmt, []).append(i)
        for (kf, vf), members in by_format.items():
            whole = PagedKVCache(head_dim, num_kv_heads, num_pages * len(members), page_tokens, kf, vf, seed=seed,
                                 norm_correction=norm_correction, rotation=rotation, device=device)
            for j, i in enumerate(members):
                self.layers[i] = PagedKVCache(head_dim, num_kv_heads, num_pages, page_tokens, kf, vf, seed=seed,
                                              norm_correction=norm_correction, rotation=rotation, device=device,
                                              k_quantizer=whole.k_quantizer, v_quantizer=whole.v_quantizer,
                                              pool=whole.pool[j * num_pages:(j + 1) * num_pages])
            self.groups.append((whole, members))
        self.num_pages = num_pages
        self.device = self.layers[0].device
        self.num_layers, self.head_dim, self.num_kv_heads = num_layers, head_dim, num_kv_heads
        self.page_tokens = page_tokens
        self._step = None

    def bytes_per_token_all_layers(self) -> int:
        return sum(layer.bytes_per_token for layer in self.layers)

    def append(self, layer: int, k, v, slot_mapping):
        self.layers[layer].append(k, v, slot_mapping)

    def attend(self, layer: int, q, block_table, seq_lens, **kw):
        return self.layers[layer].attend(q, block_table, seq_lens, **kw)

    # ------------------------------------------------------------------------------------------
    def prepare_decode(self, batch: int, num_q_heads: int, block_table, seq_lens, dtype=None):
        """Allocates the static device buffers of a decode step and captures the per-layer launches
        (append one token per sequence, attend) into one CUDA graph.  ``block_table`` must already hold
        a page for position seq_lens[b] of every sequence."""
        torch = nv.require_cuda()
        dtype = dtype or torch.float16
        dev, L, d = self.device, self.num_layers, self.head_dim
        # q, k and v of a step are three views of one buffer, so that host buffers laid out the same way
        # (host_buffers()) arrive with a single copy
        nq, nk = L * batch * num_q_heads * d, L * batch * self.num_kv_heads * d
        qkv = torch.zeros((nq + 2 * nk,), dtype=dtype, device=dev)
        st = {
            "qkv": qkv,
            "q": qkv[:nq].view(L, batch, num_q_heads, d),
            "k": qkv[nq:nq + nk].view(L, batch, self.num_kv_heads, d),
            "v": qkv[nq + nk:].view(L, batch, self.num_kv_heads, d),
            "out": torch.zeros((L, batch, num_q_heads, d), dtype=dtype, device=dev),
            "bt": block_table.to(device=dev, dtype=torch.int32).contiguous(),
            "len": seq_lens.to(device=dev, dtype=torch.int32).clone(),
            # slots of the step's new tokens, once per layer of the largest format group: layer l of a group has its
            # pages at l * num_pages in the group's pool
            "slots": torch.zeros((max(len(m) for _, m in self.groups), batch), dtype=torch.int64, device=dev),
        }
        st["workspace"] = self.layers[0].workspace(batch, num_q_heads, st["bt"].shape[1])
        st["jobs"] = self._append_jobs(0, L)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):      # warm-up outside capture (sets kernel attributes, fills caches)
            saved = st["len"].clone()
            self._slots_part(st)
            self._append_part(st, st["jobs"])
            self._attend_part(st, 0, L)
            st["len"].copy_(saved)
        torch.cuda.current_stream(dev).wait_stream(side)
        torch.cuda.synchronize(dev)
        graph = torch.cuda.CUDAGraph()
        with _capture(torch, graph):
            self._slots_part(st)
            self._append_part(st, st["jobs"])
            self._attend_part(st, 0, L)
        st["len"].copy_(saved)
        st["graph"] = graph
        st["io_streams"] = side, torch.cuda.Stream(device=dev)
        self._step = st
        return st

    # (methods that take the step's state, not closures kept in it: a cache that is dropped is then freed at once, with
    # its graphs and buffers, instead of waiting for the cyclic collector)
    def _append_jobs(self, lo, hi):
        """The append launches of layers [lo, hi), as (cache of the group, the layers' places in it, their rows): per format
        group one for each run of neighbouring layers, or a single one with its rows gathered where the group's layers are
        scattered (a launch costs less than gathering K and V)."""
        torch = nv.require_cuda()
        jobs = []
        for whole, members in self.groups:
            runs = []
            for j in (j for j, i in enumerate(members) if lo <= i < hi):      # places in the group: consecutive
                if runs and members[j] == members[j - 1] + 1:
                    runs[-1].append(j)
                else:
                    runs.append([j])
            if len(runs) <= 2:
                jobs += [(whole, slice(run[0], run[-1] + 1), slice(members[run[0]], members[run[-1]] + 1)) for run in runs]
            else:
                at = slice(runs[0][0], runs[-1][-1] + 1)
                jobs.append((whole, at, torch.tensor(members[at], device=self.device)))
        return jobs

    def _slots_part(self, st):
        """Slots of the step's new tokens, and the lengths' increment."""
        torch = nv.require_cuda()
        with torch.cuda.device(self.device):
            nv.call("tq_decode_step_slots", nv.ptr(st["bt"]), st["bt"].shape[1], nv.ptr(st["len"]), self.page_tokens,
                    st["q"].shape[1], st["slots"].shape[0], self.num_pages * self.page_tokens, nv.ptr(st["slots"]), nv.stream_ptr())

    def _append_part(self, st, jobs):
        """Quantize-on-append of the new token of the layers of ``jobs``."""
        _, batch, _, d = st["q"].shape
        for whole, at, rows in jobs:
            k, v = (t[rows] if isinstance(rows, slice) else t.index_select(0, rows) for t in (st["k"], st["v"]))
            n = (at.stop - at.start) * batch
            whole.append(k.reshape(n, self.num_kv_heads, d), v.reshape(n, self.num_kv_heads, d), st["slots"][at].reshape(-1))

    def _attend_part(self, st, lo, hi):
        for i in range(lo, hi):
            # An attention call that follows another layer's attention call may start early: that kernel writes
            # nothing this one reads before its dependency wait, and the queries and the new rows of its layer are in
            # place before the first launch of its part.  The first call of a step follows the append, which writes
            # the cache slot of the new token: it runs in stream order, in the form of the calls that follow it.
            self.layers[i].attend(st["q"][i], st["bt"], st["len"], out=st["out"][i], workspace=st["workspace"],
                                  overlap="q" if i > 0 else False, chain_head=(i == 0))

    # Parts of a step: the bytes that the first copy in and the last copy out carry, about 5 and 2.5 us of the bus --
    # what is left of the copies outside the kernels -- and the growth from one part to the next.  A layer's cache is
    # read far slower than its rows cross the bus, so that a part four times as large arrives under the one in front
    # of it; each part costs its own append launches, which is why a step below four first copies stays in one part.
    _PART_IN, _PART_OUT, _PART_GROWTH = 256 << 10, 128 << 10, 4

    @staticmethod
    def _cuts(layers, layer_bytes, first, growth):
        """Bounds of parts of ``layers`` layers, the first of at least ``first`` bytes, each ``growth`` times the last."""
        cuts, n = [0], max(1, -(-first // layer_bytes))
        while layers - cuts[-1] > n:
            cuts.append(cuts[-1] + n)
            n *= growth
        return cuts + [layers]

    def host_buffers(self):
        """Pinned host tensors (q, k, v, out) for decode_step, q/k/v carved from one allocation in the order of the
        device buffers: a step then needs one host-to-device copy instead of three."""
        torch = nv.require_cuda()
        st = self._step
        flat = torch.zeros(st["qkv"].shape, dtype=st["qkv"].dtype).pin_memory()
        nq, nk = st["q"].numel(), st["k"].numel()
        out = torch.zeros(st["out"].shape, dtype=st["out"].dtype).pin_memory()
        return (flat[:nq].view(st["q"].shape), flat[nq:nq + nk].view(st["k"].shape), flat[nq + nk:].view(st["v"].shape), out)

    def _copy_in(self, q_host, k_host, v_host):
        st = self._step
        esz = q_host.element_size()
        if (q_host.is_contiguous() and k_host.is_contiguous() and v_host.is_contiguous()
                and k_host.data_ptr() == q_host.data_ptr() + q_host.numel() * esz
                and v_host.data_ptr() == k_host.data_ptr() + k_host.numel() * esz
                and q_host.dtype == st["qkv"].dtype and q_host.numel() == st["q"].numel()):
            flat = q_host.reshape(-1).as_strided((st["qkv"].numel(),), (1,))     # the three views as one extent
            st["qkv"].copy_(flat, non_blocking=True)
        else:
            st["q"].copy_(q_host, non_blocking=True)
            st["k"].copy_(k_host, non_blocking=True)
            st["v"].copy_(v_host, non_blocking=True)

    def decode_step(self, q_host, k_host, v_host, out_host):
        """One decode step from host buffers (tensors shaped like the static device buffers): H2D of the step's
        queries and new K/V rows, the captured launches, D2H of the outputs.  With pinned buffers the copies are
        nodes of the same graph as the kernels, captured the first time a set of buffers is seen, so that a step
        is one graph launch and one synchronisation; pass the same buffers every step."""
        torch = nv.require_cuda()
        st = self._step
        hosts = (q_host, k_host, v_host, out_host)
        key = (q_host.data_ptr(), k_host.data_ptr(), v_host.data_ptr(), out_host.data_ptr())
        # (buffers seen before are known to be pinned: the query of that attribute costs microseconds per tensor)
        if st.get("io_key") == key or all(t.is_pinned() for t in hosts):
            if st.get("io_key") != key:
                graph = torch.cuda.CUDAGraph()
                (side, back), L = st["io_streams"], self.num_layers
                esz = st["qkv"].element_size()
                rows = (st["q"][0].numel() + 2 * st["k"][0].numel()) * esz
                ins = [0, L]
                if L * rows >= 4 * self._PART_IN:
                    ins = self._cuts(L, rows, self._PART_IN, self._PART_GROWTH)
                outs = [L - c for c in reversed(self._cuts(L, st["out"][0].numel() * esz, self._PART_OUT, 2))]
                if len(outs) == 2:
                    outs = sorted({0, L // 2, L})
                jobs = [self._append_jobs(lo, hi) for lo, hi in zip(ins, ins[1:])]
                with _capture(torch, graph):
                    # The copies are branches of the graph.  In: the new K/V rows of a part of the layers, their
                    # append, and their queries -- the first part's queries under its append, which needs only the rows,
                    # every further part's under the attention of the part in front.  Out: the outputs of a part
                    # leave while the next is computing.
                    main = torch.cuda.current_stream(self.device)
                    nq, nk = st["q"].numel(), st["k"].numel()
                    adjacent = (len(ins) == 2 and k_host.is_contiguous() and v_host.is_contiguous()
                                and k_host.dtype == st["qkv"].dtype and k_host.numel() == nk and v_host.numel() == nk
                                and v_host.data_ptr() == k_host.data_ptr() + nk * k_host.element_size())
                    side.wait_stream(main)
                    self._slots_part(st)
                    slots = main.record_event()
                    here = []                       # per part: what its first attention call waits for
                    for part, (lo, hi) in enumerate(zip(ins, ins[1:])):
                        with torch.cuda.stream(side):
                            if adjacent:            # rows of K and V side by side on the host (host_buffers()): one copy
                                st["qkv"][nq:].copy_(k_host.reshape(-1).as_strided((2 * nk,), (1,)), non_blocking=True)
                            else:
                                st["k"][lo:hi].copy_(k_host[lo:hi], non_blocking=True)
                                st["v"][lo:hi].copy_(v_host[lo:hi], non_blocking=True)
                            if part:
                                side.wait_event(slots)
                                self._append_part(st, jobs[part])
                        if part == 0:
                            main.wait_stream(side)
                            self._append_part(st, jobs[part])
                        with torch.cuda.stream(side):
                            # (after the append of a further part: the edge from a copy to a kernel is a full one, so
                            # that no call of the part starts before the append has completed)
                            st["q"][lo:hi].copy_(q_host[lo:hi], non_blocking=True)
                            here.append(side.record_event())
                    done = 0
                    bounds = sorted({*ins, *outs})
                    for lo, hi in zip(bounds, bounds[1:]):
                        if lo in ins:
                            main.wait_event(here[ins.index(lo)])
                        self._attend_part(st, lo, hi)
                        if hi in outs:
                            back.wait_stream(main)
                            with torch.cuda.stream(back):
                                out_host[done:hi].copy_(st["out"][done:hi], non_blocking=True)
                            done = hi
                    main.wait_stream(side)
                    main.wait_stream(back)
                st["io_graph"], st["io_key"], st["io_refs"] = graph, key, (hosts, jobs)   # the graph holds raw pointers
            st["io_graph"].replay()
        else:
            self._copy_in(q_host, k_host, v_host)
            st["graph"].replay()
            out_host.copy_(st["out"], non_blocking=True)
        torch.cuda.current_stream(self.device).synchronize()
        return out_host
