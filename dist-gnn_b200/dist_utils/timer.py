"""Keyed timers with the reference's keys and summary format (light_dist_gnn/dist_utils/timer.py:30-85).

`timing(key)` is wall clock, as in the reference.  `timing_cuda(key)` does NOT synchronise the device around the
region the way the reference does (timer.py:16-24; four host syncs per stage there): it records a pair of CUDA
events (pooled in the library) on the current stream and adds their elapsed time when a summary is asked for, so timing a region leaves
the broadcast/SpMM overlap intact.  On a CPU-only process it degrades to wall clock.
"""
import itertools
import statistics
import sys
import time
from collections import defaultdict

import torch


class TimerCtx:
    """Wall-clock region."""

    def __init__(self, timer, key):
        self.timer, self.key = timer, key

    def __enter__(self):
        self.t0 = time.time()
        return self

    def __exit__(self, *exc):
        self.timer.duration_dict[self.key] += time.time() - self.t0
        self.timer.count_dict[self.key] += 1


class CudaTimerCtx:
    """Device region between two marks of the library's event pool (spmm_cpp.mark), about 1 us each on the host."""

    def __init__(self, timer, key, mark):
        self.timer, self.key, self.mark = timer, key, mark

    def __enter__(self):
        self.begin = self.mark()
        return self

    def __exit__(self, *exc):
        timer = self.timer
        timer.pending.append((self.key, self.begin, self.mark()))
        if len(timer.pending) >= timer.MAX_PENDING:       # a long run never holds more than this many pairs
            timer.resolve()
        timer.count_dict[self.key] += 1


class DistTimer:
    MAX_PENDING = 4096
    NATIVE_KEYS = ('broadcast+spmm', 'mm', 'all_reduce')     # what the library's own regions are called
    _idents = itertools.count()

    def __init__(self, env):
        self.env = env
        self.start_time_dict = {}
        self.duration_dict = defaultdict(float)
        self.count_dict = defaultdict(int)
        self.pending = []
        self._mark = None
        self.ident = next(self._idents)

    def resolve(self, synchronize=True):
        """Adds the elapsed time of the recorded mark pairs to their keys, those of regions inside the library's calls
        included.  The training loop calls it with synchronize=False right after it has read the loss (the device is idle
        then), so the list never grows."""
        spmm_cpp = sys.modules.get('spmm_cpp')
        if spmm_cpp is None:                                # nothing was ever timed on a device
            return
        native = spmm_cpp._binding is not None and spmm_cpp._binding.pending_regions(self.ident) > 0
        if synchronize and (native or self.pending):
            torch.cuda.synchronize(self.env.device if self.env.device.type == 'cuda' else None)
        if native:
            for key, (seconds, count) in zip(self.NATIVE_KEYS, spmm_cpp._binding.resolve_regions(self.ident)):
                if count:
                    self.duration_dict[key] += seconds
                    self.count_dict[key] += count
        if self.pending:
            pending, self.pending = self.pending, []
            for key, begin, end in pending:
                self.duration_dict[key] += spmm_cpp.mark_elapsed(begin, end) / 1000.0

    def bound_regions(self):
        """Called after a library call that times regions by itself: never more than MAX_PENDING of them are kept."""
        if sys.modules['spmm_cpp']._binding.pending_regions(self.ident) >= self.MAX_PENDING:
            self.resolve()

    _resolve = resolve

    def timing(self, key):
        return TimerCtx(self, key)

    def timing_cuda(self, key):
        if self._mark is None:
            if not torch.cuda.is_available():
                return TimerCtx(self, key)
            import spmm_cpp
            self._mark = spmm_cpp.mark
        return CudaTimerCtx(self, key, self._mark)

    def empty_region(self, key):
        """Counts a region in which this layout has nothing to do (a one-rank all-reduce)."""
        self.duration_dict[key] += 0.0
        self.count_dict[key] += 1

    def start(self, key):
        self.start_time_dict[key] = time.time()
        return self.start_time_dict[key]

    def stop(self, key, *other_keys):
        d = time.time() - self.start_time_dict[key]
        for k in (key,) + tuple(key + '-' + sub for sub in other_keys):
            self.duration_dict[k] += d
            self.count_dict[k] += 1

    def summary(self):
        self._resolve()
        return '\ntimer summary:\n' + '\n'.join('%6.2fs %5d %s' % (self.duration_dict[k], self.count_dict[k], k) for k in self.duration_dict)

    def sync_duration_dicts(self):
        self._resolve()
        self.all_durations = self.env.all_gather_object(dict(self.duration_dict))

    def _stats(self):
        self.sync_duration_dicts()
        rows = {}
        for key in self.duration_dict:
            data = [d.get(key, 0.0) for d in self.all_durations]
            # the reference calls statistics.stdev, which raises with one rank (timer.py:52); report 0 instead
            rows[key] = (statistics.mean(data), statistics.stdev(data) if len(data) > 1 else 0.0, data)
        return rows

    def summary_all(self):
        rows = self._stats()
        return '\ntimer summary:\n' + '\n'.join('%6.2fs %6.2fs %5d %s' % (rows[k][0], rows[k][1], self.count_dict[k], k) for k in rows)

    def detail_all(self):
        rows = self._stats()
        return '\ntimer summary:\n' + '\n'.join(
            '%6.2fs %6.2fs %5d %s \ndetail: %s \n--------------' % (rows[k][0], rows[k][1], self.count_dict[k], k,
                                                                   ' '.join('%6.2f' % x for x in rows[k][2])) for k in rows)
