"""Host side of the persistent scheduler kernel: uploads a Schedule and
launches mdc_megakernel_launch (csrc/megakernel.cu, csrc/sched.cuh).

The device loop replaces StaticScheduler / Cursor of
mega_dsa_cp/schedule/device.py:35-129 of the reference: each block walks its
queue row, waits until every wait event's local cell holds
arity * (phase + 1), runs the task's op, then posts its notifies.  `phase` is
scalars[0]; replaying a launch only needs that scalar bumped.
"""

from __future__ import annotations

import ctypes as C
from dataclasses import dataclass

import torch

from .. import _native as N
from ..comm.buffers import SymmetricArena
from ..events.symm import EventBuffer
from .codegen import Schedule, pack_queues


@dataclass
class DeviceSchedule:
    queue: torch.Tensor     # int32 (n_ctas, row_words)
    arity: torch.Tensor     # int32 (n_events,)
    scopes: torch.Tensor    # int32 (n_events,)
    scalars: torch.Tensor   # int64: [0] phase, [1:] dynamic extents
    phase_ctl: torch.Tensor  # int64 (1,): arrival counter of the device-side phase bump
    n_ctas: int
    row_words: int
    n_events: int
    task_off: torch.Tensor | None = None   # dynamic scheduling: int32 word offset of every task in the one shared row
    dyn_ctl: torch.Tensor | None = None    # ... and its two counters (next task, finished blocks)
    n_tasks: int = 0


def task_offsets(row) -> list[int]:
    """Word offsets of the task entries of one packed queue row (format of schedule/codegen.py)."""
    offs, pos = [], 0
    while (row[pos] & 0xFF) != 0xFF:
        offs.append(pos)
        pos += 4 + ((row[pos] >> 8) & 0x3F) + ((row[pos] >> 14) & 0x3F)
    return offs


def host_words(schedule: Schedule) -> tuple[torch.Tensor, int]:
    """What a schedule has on the device, as one int32 tensor on the host: queue rows, arities, scopes; and the row length."""
    flat, row = pack_queues(schedule)
    table = lambda x: x if len(x) else [0]
    return torch.tensor(flat + table(schedule.arity) + table(schedule.scopes), dtype=torch.int32), row


def upload_schedule(schedule: Schedule, device="cuda", n_scalars: int = 8, dynamic_ctas: int | None = None, words=None) -> DeviceSchedule:
    """dynamic_ctas: the schedule was generated for ONE queue (n_ctas = 1: all tasks of the rank in dependency
    order); the kernel runs dynamic_ctas blocks that pull tasks from it with an atomic counter.
    words: host_words(schedule), from a caller that uploads one schedule several times."""
    host, row = words or host_words(schedule)
    n_ctas = queues = len(schedule.queues)
    dyn = {}
    if dynamic_ctas is not None:
        assert n_ctas == 1, "dynamic scheduling pulls from one shared queue: generate the schedule with n_ctas = 1"
        offs = task_offsets(host[:row].tolist())
        dyn = dict(task_off=torch.tensor(offs if offs else [0], dtype=torch.int32, device=device),
                   dyn_ctl=torch.zeros(2, dtype=torch.int32, device=device), n_tasks=len(offs))
        n_ctas = dynamic_ctas
    sizes = [queues * row, max(1, len(schedule.arity)), max(1, len(schedule.scopes))]
    queue, arity, scopes = host.to(device, copy=True).split(sizes)
    return DeviceSchedule(**dyn,
        queue=queue.view(queues, row), arity=arity, scopes=scopes,
        scalars=torch.zeros(n_scalars, dtype=torch.int64, device=device),
        phase_ctl=torch.zeros(1, dtype=torch.int64, device=device),
        n_ctas=n_ctas, row_words=row, n_events=schedule.n_events,
    )


def mega_params(ds: DeviceSchedule, events: EventBuffer, arena: SymmetricArena | None, status: torch.Tensor,
                log: torch.Tensor | None = None, wait_budget_ns: int = 2_000_000_000, test_off: int = 0, test_slot_bytes: int = 0,
                device_phase: bool = False) -> N.MegaParams:
    """The launch parameters of a schedule without its layer: they stay the same from step to step, so a caller
    that launches repeatedly builds them once."""
    p = N.MegaParams()
    p.queue, p.row_words, p.n_ctas = N.ptr(ds.queue), ds.row_words, ds.n_ctas
    p.scalars, p.arity, p.scopes, p.n_events = N.ptr(ds.scalars), N.ptr(ds.arity), N.ptr(ds.scopes), ds.n_events
    p.events = N.EventSetC(events.tensor.data_ptr(), events.offsets.data_ptr(), events.rank, events.world_size)
    if arena is not None:
        p.arena = N.PeerBufferC(arena.tensor.data_ptr(), arena.offsets.data_ptr(), arena.rank, arena.world_size,
                                arena.mc_base)
    else:
        p.arena = N.PeerBufferC(None, events.offsets.data_ptr(), events.rank, events.world_size, 0)
    p.wait_budget_ns = wait_budget_ns
    p.status = N.ptr(status)
    p.log = N.ptr(log)
    p.log_cap = 0 if log is None else log.numel()
    p.test_off, p.test_slot_bytes = test_off, test_slot_bytes
    p.phase_ctl = N.ptr(ds.phase_ctl) if device_phase else None
    if ds.task_off is not None:
        p.dyn_task_off, p.dyn_n_tasks, p.dyn_ctl = N.ptr(ds.task_off), ds.n_tasks, N.ptr(ds.dyn_ctl)
    return p


def launch_params(p: N.MegaParams, layer: N.LayerParams | None = None, stream=None, trace: torch.Tensor | None = None,
                  wait_budget_ns: int | None = None) -> None:
    """One launch with parameters of mega_params() (asynchronous).  `p` is only read: what belongs to this launch (the
    layer, the trace, a wait budget other than p's) goes into the launch's own copy."""
    rc = N.host().megakernel(C.addressof(p), 0 if layer is None else C.addressof(layer), None if stream is None else N.stream_ptr(stream),
                             0 if trace is None else trace.data_ptr(), 0 if trace is None else (trace.numel() - 4) // 4, wait_budget_ns)
    if rc < 0:
        N.check(rc, "mdc_megakernel_launch")


def launch_megakernel(ds: DeviceSchedule, events: EventBuffer, arena: SymmetricArena | None, status: torch.Tensor,
                      layer: N.LayerParams | None = None, log: torch.Tensor | None = None,
                      wait_budget_ns: int = 2_000_000_000, test_off: int = 0, test_slot_bytes: int = 0,
                      stream=None, trace: torch.Tensor | None = None, device_phase: bool = False) -> None:
    """One launch of the persistent kernel on this rank (asynchronous).  `trace`: optional int64
    tensor of 4 + 4 * entries words that receives the task timeline (word 0 = entry count).
    `device_phase`: the kernel itself advances scalars[0] after every block has read it (the
    reference's device-side step counter, docs/event-system.md:32-36), so the same launch can be
    replayed, also from a captured CUDA graph, with no host write in between."""
    launch_params(mega_params(ds, events, arena, status, log, wait_budget_ns, test_off, test_slot_bytes, device_phase), layer, stream,
                  trace)
