"""Run independent jobs of the solve concurrently, each on its own CUDA stream.

The Hessian factorisation and the column sweep of one module are long chains of small,
dependent kernel launches that leave most of the GPU idle; the chains of different Hessians
are independent of each other.  Each job gets a side stream; the jobs are queued by a host thread
per stream (``run_concurrent``; the C library releases the interpreter lock during its calls and
keeps its caches per thread) or all by the calling thread (``run_queued``).

Ordering contract: side streams start after everything already queued on the caller's
current stream and the caller's stream waits for every side stream before this function
returns, so callers need no extra synchronisation.  Side streams are used nowhere else,
which also makes the caching allocator's per-stream block reuse safe for tensors that are
allocated in a job and consumed by the caller afterwards.
"""
from __future__ import annotations

import os as _os
import threading
from typing import Callable, List, Sequence

import torch

_STREAMS: dict = {}
_LOCK = threading.Lock()


def _side_streams(device: torch.device, n: int) -> List["torch.cuda.Stream"]:
    with _LOCK:
        have = _STREAMS.setdefault((device.type, device.index), [])
        while len(have) < n:
            # the first stream runs the longest job: give it priority over the others
            have.append(torch.cuda.Stream(device=device, priority=(-1 if not have and _os.environ.get('B200Q_STREAM_PRIORITY', '1') == '1' else 0)))
        return have[:n]


def run_concurrent(jobs: Sequence[Callable[[], object]], device, max_streams: int = 4) -> list:
    """Call every job; returns their results in order.  Jobs are started in the order given
    (put the longest first).  The first exception raised by a job is re-raised here after all
    jobs have ended."""
    jobs = list(jobs)
    device = torch.device(device)
    if len(jobs) <= 1 or max_streams <= 1 or device.type != "cuda":
        return [job() for job in jobs]
    if device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    n = min(max_streams, len(jobs))
    streams = _side_streams(device, n)
    main = torch.cuda.current_stream(device)
    ready = torch.cuda.Event()
    ready.record(main)
    # static assignment, worker i runs jobs i, i + n, ...: the first job gets the priority stream and
    # every job meets the same stream (and its allocator pool) on every call
    results: list = [None] * len(jobs)
    errors: list = []
    grad = torch.is_grad_enabled()

    def worker(first, stream):
        torch.cuda.set_device(device)
        with torch.cuda.stream(stream), torch.set_grad_enabled(grad):
            stream.wait_event(ready)
            for i in range(first, len(jobs), n):
                try:
                    results[i] = jobs[i]()
                except BaseException as e:  # noqa: BLE001 - re-raised by the caller below
                    errors.append(e)
                    return

    threads = [threading.Thread(target=worker, args=(i, s), daemon=True) for i, s in enumerate(streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in streams:
        main.wait_stream(s)
    if errors:
        raise errors[0]
    return results


def run_queued(jobs: Sequence[Callable[[], Callable[[], object]]], device) -> list:
    """``run_concurrent`` for jobs, a stream each, that queue their work without waiting for the device and return a
    callable that waits for it and ends the job.  The calling thread queues them all (longest first), then ends them:
    with a host thread each, the jobs of a decoder layer spent as long waiting for the interpreter as queueing
    (hidden 768 / intermediate 2048: 4.9 ms, 3.2 this way; hidden 2048 / intermediate 5632, bound by the device: 6.3).
    A job that raises, when it is queued or when it is ended, keeps none of the others from being ended; the first
    exception is re-raised after that."""
    jobs = list(jobs)
    device = torch.device(device)
    if len(jobs) <= 1 or device.type != "cuda":
        return [job()() for job in jobs]
    if device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    streams = _side_streams(device, len(jobs))
    main = torch.cuda.current_stream(device)
    ready = torch.cuda.Event()
    ready.record(main)
    errors: list = []

    def attempt(stream, call):
        with torch.cuda.stream(stream):
            try:
                return call()
            except Exception as e:  # noqa: BLE001 - re-raised below
                errors.append(e)
                return None

    try:
        for stream in streams:
            stream.wait_event(ready)
        ends = [attempt(stream, job) for job, stream in zip(jobs, streams)]
        results = [None if end is None else attempt(stream, end) for end, stream in zip(ends, streams)]
    finally:
        for stream in streams:
            main.wait_stream(stream)
    if errors:
        raise errors[0]
    return results
