"""Drop-in binary_pursuit() on a B200.

Same signature, arguments, return values and side effect as
spikesorting_fullpursuit.overlap.binary_pursuit_parallel.binary_pursuit
(binary_pursuit_parallel.py:175-1532):

    binary_pursuit(voltage, v_dtype, sort_info, separability_metrics,
                   n_max_shift_inds=None, kernels_path=None, max_gpu_memory=None)
      -> (event_indices int64[n], neuron_labels int64[n],
          binary_pursuit_spike_bool bool[n], adjusted_clips)

The pursuit of each chunk runs in libfbp.so (hand-written sm_100a CUDA behind
the C ABI of include/fbp.h) on PyTorch-owned device buffers.  Chunking follows
the reference's device-memory planner with this GPU's memory, so chunk
boundaries (and the duplicate spikes the reference leaves in the 3W chunk
overlaps) are the reference's.  Results equal the reference kernels run with
their work-groups in order: where the reference's outcome depends on which
work-item runs first, the outcome of in-order execution is the one reproduced.

Differences, all documented:
* ``kernels_path`` is accepted and ignored (there is no OpenCL source).
* If the first pass of a chunk flags no window for the overlap recheck the
  reference raises UnboundLocalError (binary_pursuit_parallel.py:1369-1371
  releases buffers it never created); this implementation returns the empty
  result it was meant to return.
* The reference's pass loop has no limit (binary_pursuit_parallel.py:907);
  here a chunk that still adds spikes after ``max_passes`` passes raises
  FbpError (status FBP_E_PASSES) instead of running on.
* Keyword-only extras: ``mode`` ("fast": likelihood by transforms and screened
  overlap recheck, both exact; "plain": scalar FP32 kernels), ``device``,
  ``work_group_size`` (the reference's kernel work-group size, 256, whose
  execution order the results follow), ``max_passes``,
  ``dedupe_chunk_seams`` (drop a chunk's spikes that the previous chunk found
  with the same index and label in their 3-window overlap; off by default,
  where the output is the reference's, duplicates included), ``tuning``
  (launch shapes: None for the library's, "auto" to measure them on the first
  chunk with spikesorting_fullpursuit_b200.autotune, or a dict), ``verbose``,
  ``return_stats``.
"""
from __future__ import annotations

import ctypes
import os
import threading
from concurrent.futures import ThreadPoolExecutor

import numpy as np

from .. import _native, autotune
from ..processing.conversions import time_window_to_samples

WORK_GROUP_SIZE = 256
MAX_PASSES = _native.MAX_PASSES   # default pass limit of one chunk
MAX_CAPACITY_RETRIES = 4   # re-runs of a chunk whose spikes outgrew the output buffers
CAPACITY_PER_WINDOW = 16   # spike slots of a chunk's first attempt, per window ...
CAPACITY_EXTRA = 1024      # ... plus these


def plan_chunks(n_samples, n_chans, n_templates, template_samples_per_chan, sampling_rate,
                n_max_shift_inds, global_mem_size, max_gpu_memory=None,
                work_group_size=WORK_GROUP_SIZE, address_bits=64):
    """Chunk onsets and chunk length from the device-memory budget.

    Follows binary_pursuit_parallel.py:389-475 (budget per second of data:
    voltage, likelihood, per-window buffers and the overlap group buffers) and
    :498-507 (onsets overlap by 3 windows).  Arithmetic types follow the
    reference so the floor() lands on the same sample count."""
    W = int(template_samples_per_chan)
    budget = max(global_mem_size * 0.5, global_mem_size - (1024 * 1024 * 1024))
    if max_gpu_memory is not None:
        budget = min(budget, max_gpu_memory)
    assert budget > 0
    S = int(n_max_shift_inds)
    items = np.int64((2 * S + 1) * (2 * S + 1) * n_templates)
    groups = np.int64(((items - 1) / np.int64(work_group_size)) + 1)
    fixed = n_templates * n_chans * W * 4 + n_templates * 4
    chans = np.uint32(n_chans)
    per_second = chans * sampling_rate * 4
    per_second += n_templates * sampling_rate * 4
    per_second += (sampling_rate / W) * (5 * 4 + (groups / 3) * 4 + (groups / 3) * 4)
    seconds = (budget - fixed) / per_second
    seconds = min(seconds, np.floor(((1 << address_bits) - 1) / (4 * sampling_rate * chans)))
    chunk = int(np.floor(seconds * sampling_rate))
    if chunk < 4 * W:
        raise ValueError("Cannot fit enough data on GPU to run binary pursuit. "
                         "Decrease template samples or get a new GPU.")
    onsets = []
    onset = 0
    while onset < n_samples - W:
        onsets.append(onset)
        onset += chunk - 3 * W
    return onsets, chunk


def seam_duplicates(prev_idx, prev_lab, idx, lab, seam_start):
    """Which of a chunk's spikes the previous chunk already found.

    Chunks overlap by 3 windows (binary_pursuit_parallel.py:498-507) and the
    reference keeps the spikes both chunks find in the overlap
    (binary_pursuit_parallel.py:1491, left to later post-processing).  A spike of
    this chunk at or after ``seam_start`` (the chunk's onset) is a duplicate when
    the previous chunk has a spike with the same index and label.  Indices are
    absolute sample indices; returns a boolean mask over ``idx``."""
    idx = np.asarray(idx, dtype=np.int64)
    lab = np.asarray(lab, dtype=np.int64)
    prev_idx = np.asarray(prev_idx, dtype=np.int64)
    prev_lab = np.asarray(prev_lab, dtype=np.int64)
    dup = np.zeros(idx.size, dtype=bool)
    if idx.size == 0 or prev_idx.size == 0:
        return dup
    sel = prev_idx >= seam_start
    width = int(max(lab.max(initial=0), prev_lab.max(initial=0))) + 1
    prev_keys = np.unique(prev_idx[sel] * width + prev_lab[sel])
    mine = idx >= seam_start
    dup[mine] = np.isin(idx[mine] * width + lab[mine], prev_keys, assume_unique=False)
    return dup


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class _Uploader:
    """Host -> device copy of voltage chunks.

    Short float32 chunks go as they are (``direct``).  Others go in blocks of some
    samples of every channel: host threads convert and copy blocks into page-locked
    slabs, each as soon as a slab is free, while the copy engine moves the earlier
    blocks to the device on a stream of its own.  The source may be any real dtype and
    any row-strided view: the float32 conversion happens in the slab copy.

    Blocks of all channels keep both sides busy from the first one on: with a slab
    per 2M samples of one channel, 16 of them filled before the first was sent,
    16 channels x 120 s took 12.4 ms to upload, as here 9.0 ms."""

    # 307 MB with 4 / 8 / 16 threads: slabs of 4 MB 11.6 / 9.0 / 11.4 ms, of 8 MB 12.8 / 9.7 /
    # 10.8 ms, of 2 MB 11.0 / 12.3 / 16.1 ms; 8 to 32 slabs differ by less than 10%
    SLAB_FLOATS = 1 << 20    # 4 MB per slab ...
    LEAST_FLOATS = 1 << 19   # ... and less where a chunk has fewer than 16 of those, down to 2 MB
    N_SLABS = 16
    N_THREADS = max(1, min(8, os.cpu_count() or 2))
    # Pageable memory goes at about 20 GB/s, read by the calling thread; slabs are faster
    # once their threads run: 3.2 MB 0.2 (slabs 0.9), 38 MB 1.8 (3.4), 77 MB 5.4 (4.3) ms
    DIRECT_BYTES = 48 << 20

    def __init__(self, torch, dev):
        self.torch = torch
        self.dev = dev
        self.stream = None
        self.pool = None

    def direct(self, host, dst):
        """Upload a short chunk on the caller's stream; False if the chunk is not one."""
        C, N = host.shape
        if not (isinstance(host, np.ndarray) and host.dtype == np.float32 and 4 * C * N <= self.DIRECT_BYTES
                and host.strides[1] == 4 and (C == 1 or host.strides[0] >= 4 * N)):
            return False
        stream = ctypes.c_void_p(self.torch.cuda.current_stream(self.dev).cuda_stream)
        with self.torch.cuda.device(self.dev):
            _native.check(_native.lib().fbp_copy_rows(_ptr(dst), 4 * dst.stride(0), ctypes.c_void_p(host.ctypes.data),
                                                      host.strides[0] if C > 1 else 4 * N, 4 * N, C, stream))
        return True

    def upload(self, host, dst):
        """Upload ``host``; the caller's stream waits for it."""
        if not self.direct(host, dst):
            self.start_staged(host, dst)[3]()

    def start_staged(self, host, dst):
        """Upload ``host`` on host threads, time range by time range.

        Returns (events, upto, flags, finish): events[k] completes once samples
        [0, upto[k]) of every channel are in ``dst``; flags[k] turns 1 once events[k]
        is recorded (the library waits for it before waiting on the event);
        ``finish()`` joins the thread and re-raises its error, if any.  After an error the
        rest of ``dst`` is zero: a pursuit already behind the upload finds nothing there."""
        torch = self.torch
        C, N = host.shape
        slab = min(self.SLAB_FLOATS, max(self.LEAST_FLOATS, -(-C * N // 16)))
        span = max(1, slab // C)
        ranges = [(a, min(N, a + span)) for a in range(0, N, span)]
        n_slabs = min(self.N_SLABS, len(ranges))
        slabs = [torch.empty(C * span, dtype=torch.float32, pin_memory=True) for _ in range(n_slabs)]
        if self.pool is None:
            self.stream = torch.cuda.Stream(self.dev)
            self.pool = ThreadPoolExecutor(self.N_THREADS)
        stream, pool = self.stream, self.pool
        events = [torch.cuda.Event() for _ in ranges]
        flags = np.zeros(len(ranges), dtype=np.uint32)
        upto = np.array([b for _, b in ranges], dtype=np.uint32)
        stream.wait_stream(torch.cuda.current_stream(self.dev))   # dst may still be read by earlier work
        for ev in events:   # creates the CUDA events (torch makes them at the first record)
            ev.record(stream)
        copy_rows, handle = _native.lib().fbp_copy_rows, ctypes.c_void_p(stream.cuda_stream)
        failure = []

        def fill(k):
            if k >= n_slabs:
                events[k - n_slabs].synchronize()   # the slab's previous block has left it
            a, b = ranges[k]
            np.copyto(slabs[k % n_slabs].numpy()[:C * (b - a)].reshape(C, b - a), host[:, a:b], casting="unsafe")

        def run():
            try:
                with torch.cuda.device(self.dev):
                    filled = [pool.submit(fill, k) for k in range(n_slabs)]
                    for k, (a, b) in enumerate(ranges):
                        filled[k].result()
                        width = 4 * (b - a)
                        _native.check(copy_rows(ctypes.c_void_p(dst.data_ptr() + 4 * a), 4 * dst.stride(0),
                                                _ptr(slabs[k % n_slabs]), width, width, C, handle))
                        events[k].record(stream)
                        flags[k] = 1
                        if k + n_slabs < len(ranges):
                            filled.append(pool.submit(fill, k + n_slabs))
            except BaseException as e:   # the library must not wait for ranges that never come
                failure.append(e)
                with torch.cuda.device(self.dev), torch.cuda.stream(stream):
                    k0 = int(np.count_nonzero(flags))   # flags turn 1 in order
                    try:
                        if k0 < len(ranges):
                            dst[:, ranges[k0][0]:].zero_()
                    finally:
                        for k in range(k0, len(ranges)):
                            events[k].record(stream)
                            flags[k] = 1
            finally:   # the slabs go back to torch's pinned cache: their last copies must be done
                stream.synchronize()

        th = threading.Thread(target=run, daemon=True)
        th.start()

        def finish():
            th.join()
            torch.cuda.current_stream(self.dev).wait_stream(stream)
            if failure:
                raise failure[0]

        return events, upto, flags, finish

    def close(self):
        if self.pool is not None:
            self.pool.shutdown(wait=True)


class _Pursuer:
    """Device buffers and the C-ABI calls for one binary_pursuit() call."""

    def __init__(self, torch, dev, n_chans, templates, bias, theta, W, S, max_chunk, flags,
                 work_group_size, max_passes, tuning=None):
        self.torch = torch
        self.dev = dev
        self.C, self.W, self.S = n_chans, W, S
        self.M = templates.shape[0]
        self.flags = flags
        self.wg = work_group_size
        self.max_passes = int(max_passes)
        # templates, bias and thresholds in one copy, each part 256-byte aligned
        parts = [np.ravel(x).astype(np.float32, copy=False) for x in (templates, bias, theta)]
        at = np.cumsum([0] + [-(-x.size // 64) * 64 for x in parts])
        flat = np.zeros(at[-1], dtype=np.float32)
        for x, o in zip(parts, at):
            flat[o:o + x.size] = x
        flat = torch.from_numpy(flat).to(dev)
        self.T, self.bias, self.theta = (flat[o:o + x.size] for x, o in zip(parts, at))
        self.T = self.T.view(templates.shape)
        d = _native.dims(n_chans, max_chunk, self.M, W, S, work_group_size)
        nbytes = _native.workspace_bytes(d, flags)
        if nbytes == 0:
            raise ValueError("invalid binary pursuit sizes for the GPU library")
        self.ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        self.V = torch.empty((n_chans, max_chunk), dtype=torch.float32, device=dev)
        self.up = _Uploader(torch, dev)
        self.tuning = tuning
        self.stats = []

    def chunk(self, host_chunk, clips):
        """Pursue one chunk (``host_chunk``: C x N view of the caller's voltage)."""
        torch = self.torch
        C, N = host_chunk.shape
        d = _native.dims(C, N, self.M, self.W, self.S, self.wg)
        V = self.V[:, :N] if N == self.V.shape[1] else self.V.view(-1)[:C * N].view(C, N)
        # the first pass runs behind the upload unless the chunk is short or the autotuner
        # must see the voltage first
        ready = None
        if self.tuning == "auto":
            self.up.upload(host_chunk, V)
        elif not self.up.direct(host_chunk, V):
            ready = self.up.start_staged(host_chunk, V)
        nw = (N + self.W - 1) // self.W
        # every pass adds at most one spike per window; dense probes end with about five
        # spikes per window, so the first attempt holds 16 (8 B each, far below the
        # likelihood's 4*M*W bytes per window) and a capacity retry, which pursues the
        # chunk again, stays rare
        most = nw * self.max_passes if self.max_passes > 0 else 0xFFFFFFFF
        cap = min(CAPACITY_PER_WINDOW * nw + CAPACITY_EXTRA, most, 0xFFFFFFFF)
        stream = ctypes.c_void_p(torch.cuda.current_stream(self.dev).cuda_stream)
        L = _native.lib()
        if self.tuning == "auto":
            self.tuning = autotune.tune(V, self.T.cpu().numpy(), self.bias.cpu().numpy(), self.theta.cpu().numpy(),
                                        self.W, self.S, overlap=bool(self.flags & _native.FBP_OVERLAP_RECHECK),
                                        device=self.dev)
        autotune.apply(self.tuning)
        try:
            return self._pursue(host_chunk, clips, V, d, N, nw, most, cap, stream, L, ready)
        finally:
            autotune.apply(None)

    def _pursue(self, host_chunk, clips, V, d, N, nw, most, cap, stream, L, ready=None):
        torch = self.torch
        C = V.shape[0]
        for attempt in range(MAX_CAPACITY_RETRIES + 1):
            idx = torch.empty(cap, dtype=torch.int32, device=self.dev)
            lab = torch.empty(cap, dtype=torch.int32, device=self.dev)
            n = ctypes.c_uint32(0)
            st = _native.FbpChunkStats()
            if ready is not None:
                events, upto, flags, finish = ready
                ready = None
                evp = (ctypes.c_void_p * len(events))(*[e.cuda_event for e in events])
                try:
                    rc = L.fbp_pursue_chunk_staged(ctypes.byref(d), self.flags, _ptr(V), _ptr(self.T),
                                                   _ptr(self.bias), _ptr(self.theta), _ptr(self.ws),
                                                   self.ws.numel(), _ptr(idx), _ptr(lab), cap, ctypes.byref(n),
                                                   ctypes.byref(st), self.max_passes, evp,
                                                   upto.ctypes.data_as(ctypes.c_void_p),
                                                   flags.ctypes.data_as(ctypes.c_void_p), len(events), stream)
                finally:
                    finish()
            else:
                rc = L.fbp_pursue_chunk(ctypes.byref(d), self.flags, _ptr(V), _ptr(self.T),
                                        _ptr(self.bias), _ptr(self.theta), _ptr(self.ws),
                                        self.ws.numel(), _ptr(idx), _ptr(lab), cap, ctypes.byref(n),
                                        ctypes.byref(st), self.max_passes, stream)
            if rc != _native.FBP_E_CAPACITY:
                break
            if cap >= min(most, 0xFFFFFFFF) or attempt == MAX_CAPACITY_RETRIES:
                _native.check(rc)
            # n holds a lower bound of what the chunk needs; the voltage was partly pursued
            cap = int(min(max(4 * cap, 2 * n.value), most, 0xFFFFFFFF))
            self.up.upload(host_chunk, V)
        self.stats.append(st.as_dict())
        _native.check(rc)
        k = n.value
        out_clips = []
        if clips and k > 0:
            cl = torch.zeros((k, C * self.W), dtype=torch.float32, device=self.dev)
            _native.check(L.fbp_adjusted_clips(ctypes.byref(d), _ptr(V), _ptr(self.T), _ptr(idx),
                                               _ptr(lab), k, _ptr(cl), stream))
            out_clips = cl.cpu().numpy()
        si = idx[:k].cpu().numpy().view(np.uint32)
        sl = lab[:k].cpu().numpy().view(np.uint32)
        return si, sl, out_clips

    def close(self):
        self.up.close()


def binary_pursuit(voltage, v_dtype, sort_info, separability_metrics, n_max_shift_inds=None,
                   kernels_path=None, max_gpu_memory=None, *, mode="fast", device=None,
                   work_group_size=WORK_GROUP_SIZE, max_passes=MAX_PASSES,
                   dedupe_chunk_seams=False, tuning=None, verbose=True, return_stats=False):
    """Find template spikes in ``voltage`` by binary pursuit on the GPU.

    See the module docstring for the contract; the arguments mean what they
    mean for the reference function (binary_pursuit_parallel.py:175-183)."""
    import torch

    del kernels_path
    if not torch.cuda.is_available():
        raise RuntimeError("No GPU available")
    _native.lib()
    dev = (device if isinstance(device, torch.device)
           else torch.device("cuda", torch.cuda.current_device() if device is None else int(device)))
    n_chans = int(voltage.shape[0])
    n_samples = int(voltage.shape[1])
    sampling_rate = sort_info["sampling_rate"]
    chan_win, _ = time_window_to_samples(sort_info["clip_width"], sampling_rate)
    W = int(sort_info["n_samples_per_chan"])
    templates = separability_metrics["templates"]
    if templates.ndim == 1:
        templates = np.reshape(templates, (1, -1))
    templates = np.float32(templates)
    M = templates.shape[0]
    clip_init_samples = int(np.abs(chan_win[0]))
    bias = np.float32(-0.5 * separability_metrics["template_SS"])
    theta = np.float32(separability_metrics["neuron_lower_thresholds"])
    if n_max_shift_inds is None or n_max_shift_inds < 0:
        n_max_shift_inds = W // 2
    S = int(np.uint32(n_max_shift_inds))
    total_mem = torch.cuda.get_device_properties(dev).total_memory
    onsets, chunk_len = plan_chunks(n_samples, n_chans, M, W, sampling_rate, S, total_mem,
                                    max_gpu_memory, work_group_size)
    flags = _native.FBP_OVERLAP_RECHECK if sort_info["do_overlap_recheck"] else 0
    if mode == "plain":
        flags |= _native.FBP_PLAIN_FP32
    elif mode != "fast":
        raise ValueError("mode must be 'fast' or 'plain'")
    get_clips = bool(sort_info["get_adjusted_clips"])
    idx_all, lab_all, bool_all, clips_all = [], [], [], []
    pursuer = None
    if onsets:
        max_chunk = min(n_samples, chunk_len)
        pursuer = _Pursuer(torch, dev, n_chans, templates, bias, theta, W, S, max_chunk, flags,
                           work_group_size, max_passes, tuning)
    try:
        for start in onsets:
            stop = int(np.uint32(min(n_samples, start + chunk_len)))
            si, sl, clips = pursuer.chunk(voltage[:, start:stop], get_clips)
            if si.size == 0:
                continue
            ab = si.astype(np.int64) + start
            if dedupe_chunk_seams and idx_all:
                keep = ~seam_duplicates(idx_all[-1], lab_all[-1], ab, sl, start)
                ab, sl = ab[keep], sl[keep]
                if get_clips and len(clips):
                    clips = clips[keep]
                if ab.size == 0:
                    continue
            idx_all.append(ab)
            lab_all.append(sl)
            clips_all.append(clips)
            bool_all.append(np.ones(ab.size, dtype=bool))
    finally:
        if pursuer is not None:
            pursuer.close()
    if idx_all:
        event_indices = np.int64(np.hstack(idx_all))
        neuron_labels = np.int64(np.hstack(lab_all))
        # one chunk's clips are already an array of the caller's own
        adjusted_clips = clips_all[0] if len(clips_all) == 1 else np.vstack(clips_all)
        adjusted_clips = np.atleast_2d(adjusted_clips).astype(v_dtype, copy=False)
        spike_bool = np.hstack(bool_all)
        event_indices += clip_init_samples
        if verbose:
            print("Found a total of", np.count_nonzero(spike_bool), "secret spikes", flush=True)
    else:
        event_indices, neuron_labels, spike_bool, adjusted_clips = [], [], [], []
        if verbose:
            print("Found a total of ZERO secret spikes", flush=True)
    # side effect of add_n_spikes (neuron_separability.py:334-345)
    labels_arr = np.asarray(neuron_labels, dtype=np.int64)
    counts = np.bincount(labels_arr, minlength=M)[:M] if labels_arr.size else np.zeros(M, dtype=np.int64)
    separability_metrics["n_spikes"] = counts.astype(np.float64)
    out = (event_indices, neuron_labels, spike_bool, adjusted_clips)
    if return_stats:
        return out, (pursuer.stats if pursuer else [])
    return out
