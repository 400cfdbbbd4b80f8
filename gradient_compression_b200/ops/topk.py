"""Batched exact Top-K selection by magnitude over many segments of one flat buffer (``csrc/gc_topk.cu``).

``TopKSelector(segments, device)`` holds the scratch state; ``select(g, e)`` returns the (global int32 index, value) lists of
all segments back to back (segment i's entries start at ``offsets[i]``), after folding the error memory ``e`` into the
selection and updating it in place: ``e <- g + e`` with the selected entries zeroed (reference: reducer.py:1161-1189).
On CPU the same contract is met with ``torch.topk`` per segment.
"""
from __future__ import annotations

import torch

from . import _native as nat


class TopKScratch:
    """Histograms and candidate lists of the selection kernels for groups of the given lengths."""

    def __init__(self, lengths, device):
        lib = nat.cuda()
        self.state = torch.zeros(lib.gc_cuda_topk_state_bytes(len(lengths)), dtype=torch.uint8, device=device)
        self.lists = torch.empty(sum(lib.gc_cuda_topk_list_bytes(n) for n in lengths), dtype=torch.uint8, device=device)


class TopKSelector:
    def __init__(self, segments, device):
        """segments: list of (start, length, k) in elements of the flat buffer."""
        self.device = torch.device(device)
        self.segments = [(int(s), int(l), int(min(k, l))) for s, l, k in segments]
        self.offsets, off = [], 0
        for _, _, k in self.segments:
            self.offsets.append(off)
            off += k
        self.total = off
        if self.device.type == "cuda":
            # runs of consecutive segments, as many as one launch takes
            most, runs = nat.cuda().gc_cuda_topk_max_segs(), []
            for i, (s, l, k) in enumerate(self.segments):
                if l == 0:
                    continue
                if not runs or len(runs[-1]) == most or self.segments[runs[-1][-1]][0] + self.segments[runs[-1][-1]][1] != s:
                    runs.append([])
                runs[-1].append(i)
            self._runs = [(r, TopKScratch([self.segments[i][1] for i in r], self.device),
                           torch.tensor([self.segments[i][2] for i in r], dtype=torch.int64)) for r in runs]

    def select(self, g, e=None, out_idx=None, out_val=None):
        g = g.contiguous().view(-1)
        if out_idx is None:
            out_idx = torch.empty(self.total, dtype=torch.int32, device=g.device)
        if out_val is None:
            out_val = torch.empty(self.total, dtype=torch.float32, device=g.device)
        if g.is_cuda:
            if e is not None and e.device != g.device:
                raise ValueError(f"values on {g.device}, error memory on {e.device}")
            with torch.cuda.device(g.device):
                for run, scratch, counts in self._runs:
                    table = (nat.SegDesc * len(run))(*[(g.data_ptr() + 4 * self.segments[i][0], None, self.segments[i][0]) for i in run])
                    off = self.offsets[run[0]]
                    nat.check(nat.cuda().gc_cuda_topk_run(table, len(run), self.segments[run[-1]][0] + self.segments[run[-1]][1], counts.data_ptr(), 1,
                                                          nat.ptr(e), scratch.state.data_ptr(), scratch.lists.data_ptr(),
                                                          out_idx.data_ptr() + 4 * off, out_val.data_ptr() + 4 * off, nat.stream_ptr()), "topk_run")
                    nat.count_launch(3)
            return out_idx, out_val
        a = g if e is None else e.add_(g)
        for (s, l, k), o in zip(self.segments, self.offsets):
            seg = a[s:s + l]
            pos = torch.topk(seg.abs(), k, sorted=False)[1]
            out_idx[o:o + k] = (pos + s).to(torch.int32)
            out_val[o:o + k] = seg[pos]
        if e is not None:
            e[out_idx.long()] = 0.0
        return out_idx, out_val
