"""All-reduce of HOST-memory gradient sets through the GPUs.

The reference reduces host buffers over TCP
(src/stdml/collective/session.cpp:64-111).  Here a pinned host buffer is cut
into chunks and each chunk flows host -> device (copy engine) -> fused
all-reduce kernel over NVLink -> host, with the three stages of different
chunks overlapped on three streams.  The device side is zero-copy: chunks land
directly in the symmetric heap and are reduced in place.
"""
import ctypes

import torch

from .. import _native
from ..ops.device import dtype_code, op_code


def piece_bounds(numel, itemsize, chunks, align=4096):
    """Where the pieces of a pipelined transfer start and end.

    While the first piece comes in, nothing goes out, and the other way round for the last
    one: pieces grow from an eighth of the middle ones and shrink back at the end, so
    that these two stretches are short (102 MB both ways: 2.54 ms with 16 equal
    pieces, 2.45 ms so; the rest is PCIe in both directions at once).  Below 2 MB per piece the launches of a piece cost
    more than its overlap gives: fewer pieces, at most `chunks`."""
    n = max(1, min(chunks, numel * itemsize // (2 << 20)))
    ramp = 3 if n >= 8 else 2 if n >= 5 else 1 if n >= 3 else 0
    weight = [2.0 ** min(0, min(i, n - 1 - i) - ramp) for i in range(n)]
    bounds, acc = [0], 0.0
    for w in weight[:-1]:
        acc += w
        at = int(round(numel * acc / sum(weight) / align)) * align
        if bounds[-1] < at < numel:
            bounds.append(at)
    return bounds + [numel]


class HostAllReduce:
    def __init__(self, sess, numel, dtype=torch.float32, chunks=8):
        if sess.vranks != 1:
            raise ValueError("HostAllReduce needs a real (one GPU per process) session")
        self.sess = sess
        self.numel = numel
        self.dtype = dtype
        self.flat = sess.symm_empty(numel, dtype)
        at = piece_bounds(numel, self.flat.element_size(), chunks)
        self.bounds = list(zip(at[:-1], at[1:]))
        self._bounds = (ctypes.c_ulonglong * len(at))(*at)
        dev = sess.device
        self.h2d = torch.cuda.Stream(dev)
        self.comm = torch.cuda.Stream(dev)
        self.d2h = torch.cuda.Stream(dev)
        self.launches_per_run = len(self.bounds)

    @property
    def h2d_bytes(self):
        return self.numel * self.flat.element_size()

    d2h_bytes = h2d_bytes

    def run(self, host_in, host_out, op="sum", scale=None):
        """host_out = scale * all_reduce(host_in); both pinned, flat, `numel` long.
        Returns when host_out is complete."""
        for name, t in (("host_in", host_in), ("host_out", host_out)):
            if t.is_cuda or t.dtype != self.dtype or t.numel() != self.numel or not t.is_contiguous():
                raise ValueError(f"HostAllReduce.run: {name} must be a contiguous host tensor of "
                                 f"{self.numel} x {self.dtype}")
            if not t.is_pinned():
                raise ValueError(f"HostAllReduce.run: {name} must be pinned (a pageable buffer "
                                 "makes every copy synchronous and ends the overlap)")
        if self.numel == 0:
            return host_out
        # pieces, events and copies are native work: in Python a piece cost 35 us of it
        _native.check(_native.lib().stdmlc_dw_host_all_reduce(
            self.sess._h, host_in.data_ptr(), host_out.data_ptr(), self.flat.data_ptr(),
            len(self.bounds), self._bounds, dtype_code(self.dtype), op_code(op),
            1.0 if scale is None else float(scale),
            torch.cuda.current_stream(self.sess.device).cuda_stream, self.h2d.cuda_stream,
            self.comm.cuda_stream, self.d2h.cuda_stream))
        return host_out

    def close(self):
        self.sess.symm_free(self.flat)
