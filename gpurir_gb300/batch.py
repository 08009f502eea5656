"""Batched simulation of many rooms in one persistent launch.

gpuRIR simulates one room per call (src/gpuRIR_cuda.cu:766); a batch of
rooms of uneven size, image counts, lengths and source/receiver counts runs
here as one launch whose work items (RIR segments) are ordered largest first.
Output is one flat float32 device array, packed room after room; room r's RIRs
are ``out[offsets[r]:offsets[r+1]].view(n_src, n_rcv, n_samples)``.

A room is a dict with simulateRIR's argument names: room_sz, beta, pos_src,
pos_rcv, nb_img, Tmax, Tdiff (optional), spkr_pattern, mic_pattern, orV_src,
orV_rcv.  All rooms of a batch share fs and c.
"""
import ctypes

import numpy as np

from . import _lib, polar_patterns, simulator


_ROOM = np.dtype(_lib.Room)


def _rows(v):
    v = np.asarray(v, dtype=np.float32)
    return v if v.ndim == 2 and v.shape[1] == 3 else v.reshape(-1, 3)


def _tables(rooms):
    """The room table and the float32 rows of every room's sources and receivers.  Each
    argument is looked at once and the table filled by columns: entry by entry, twice over,
    a batch's packing took longer than its kernels (24 rooms: 500 us a call, now 290)."""
    table = (_lib.Room * len(rooms))()
    src, rcv = [_rows(r["pos_src"]) for r in rooms], [_rows(r["pos_rcv"]) for r in rooms]
    if len(rooms):
        t = np.frombuffer(table, dtype=_ROOM)
        f32 = np.float32
        t["room_sz"] = np.concatenate([np.asarray(r["room_sz"], dtype=f32).reshape(1, 3) for r in rooms])
        t["beta"] = np.concatenate([np.asarray(r["beta"], dtype=f32).reshape(1, 6) for r in rooms])
        t["nb_img"] = [[int(x) for x in np.asarray(r["nb_img"]).reshape(3).tolist()] for r in rooms]
        t["Tmax"] = [float(r["Tmax"]) for r in rooms]
        t["Tdiff"] = [float(r["Tmax"] if r.get("Tdiff") is None else r["Tdiff"]) for r in rooms]
        t["n_src"] = [len(v) for v in src]
        t["n_rcv"] = [len(v) for v in rcv]
        t["spkr_pattern"] = [polar_patterns[r.get("spkr_pattern") or "omni"] for r in rooms]
        t["mic_pattern"] = [polar_patterns[r.get("mic_pattern") or "omni"] for r in rooms]
    return table, src, rcv


def _room_struct(rooms):
    return _tables(rooms)[0]


def _points(rooms, src, rcv):
    """Positions and orientations of all rooms in one float32 array, and the views of its
    four sections (each on a 256-byte boundary, as arrays of their own would be)."""
    n_src, n_rcv = sum(map(len, src)), sum(map(len, rcv))
    a, b = (3 * n_src + 63) // 64 * 64, (3 * n_rcv + 63) // 64 * 64
    flat = np.zeros(2 * (a + b), np.float32)
    views = []
    for at, n in ((0, n_src), (a, n_rcv), (a + b, n_src), (2 * a + b, n_rcv)):
        views.append(flat[at:at + 3 * n].reshape(n, 3))
    np.concatenate(src, out=views[0])
    np.concatenate(rcv, out=views[1])
    for key, rows, view in (("orV_src", src, views[2]), ("orV_rcv", rcv, views[3])):
        i = 0
        for r, v in zip(rooms, rows):
            if r.get(key) is not None:
                view[i:i + len(v)] = np.asarray(r[key], dtype=np.float32).reshape(len(v), 3)
            i += len(v)
    return flat, views


def pack(rooms):
    """Host arrays of a batch: (room table, pos_src, pos_rcv, orV_src, orV_rcv)."""
    table, src, rcv = _tables(rooms)
    return (table, *_points(rooms, src, rcv)[1])


def _offsets(table, fs):
    off = (ctypes.c_longlong * (len(table) + 1))()
    L = _lib.load()
    _lib.check(L.gpurir_batch_layout(len(table), table, float(fs), off), "gpurir_batch_layout")
    return np.array(off[:], dtype=np.int64)


def layout(rooms, fs):
    """Element offsets of each room's RIRs in the packed output (n_rooms + 1 values)."""
    return _offsets(_room_struct(rooms), fs)


def shapes(rooms, fs):
    from .workloads import n_samples
    return [(np.asarray(r["pos_src"]).reshape(-1, 3).shape[0],
             np.asarray(r["pos_rcv"]).reshape(-1, 3).shape[0],
             n_samples(r["Tmax"], fs)) for r in rooms]


def unpack(flat, rooms, fs):
    """Views [n_src, n_rcv, n_samples] of each room in the packed output."""
    off = layout(rooms, fs)
    return [flat[off[i]:off[i + 1]].reshape(sh) for i, sh in enumerate(shapes(rooms, fs))]


def simulate_batch(rooms, fs, c=343.0, sim=None, stream=None):
    """Simulate every room in one launch.  Returns (packed float32 CUDA tensor, offsets)."""
    import torch
    sim = sim or simulator()
    table, src, rcv = _tables(rooms)
    off = _offsets(table, fs)
    flat, views = _points(rooms, src, rcv)
    dev = torch.device("cuda", torch.cuda.current_device())
    points = torch.from_numpy(flat).to(dev)   # one upload
    at = [points.data_ptr() + v.ctypes.data - flat.ctypes.data for v in views]
    out = torch.empty(int(off[-1]), dtype=torch.float32, device=dev)
    st = stream if stream is not None else torch.cuda.current_stream().cuda_stream
    L = _lib.load()
    _lib.check(L.gpurir_simulate_batch_device(sim.handle, len(rooms), table, float(fs), float(c),
                                              *at, out.data_ptr(), ctypes.c_void_p(st)),
               "gpurir_simulate_batch_device")
    return out, off


class BatchPlan:
    """A batch planned once and captured in a CUDA graph; ``launch()`` replays it.

    The device arrays ``pos_src``, ``pos_rcv``, ``orV_src``, ``orV_rcv`` (torch
    tensors) are read at every replay: update them in place to move sources
    and receivers.  ``out`` is the packed output; ``rirs()`` gives per-room views.
    Each replay draws the next diffuse-tail noise of the simulator's seed.
    """

    def __init__(self, rooms, fs, c=343.0, sim=None):
        import torch
        self.sim = sim or simulator()
        self.rooms, self.fs = rooms, fs
        table, ps, pr, os_, or_ = pack(rooms)
        self.offsets = _offsets(table, fs)
        dev = torch.device("cuda", torch.cuda.current_device())
        self.pos_src, self.pos_rcv, self.orV_src, self.orV_rcv = \
            [torch.from_numpy(a).to(dev) for a in (ps, pr, os_, or_)]
        self.out = torch.zeros(int(self.offsets[-1]), dtype=torch.float32, device=dev)
        self._L = _lib.load()
        h = ctypes.c_void_p()
        _lib.check(self._L.gpurir_batch_create(
            self.sim.handle, len(rooms), table, float(fs), float(c), self.pos_src.data_ptr(),
            self.pos_rcv.data_ptr(), self.orV_src.data_ptr(), self.orV_rcv.data_ptr(),
            self.out.data_ptr(), ctypes.byref(h)), "gpurir_batch_create")
        self._h = h

    def launch(self, stream=None):
        import torch
        st = stream if stream is not None else torch.cuda.current_stream().cuda_stream
        _lib.check(self._L.gpurir_batch_launch(self._h, ctypes.c_void_p(st)), "gpurir_batch_launch")
        return self.out

    def rirs(self):
        return [self.out[self.offsets[i]:self.offsets[i + 1]].view(*sh)
                for i, sh in enumerate(shapes(self.rooms, self.fs))]

    def __del__(self):
        L, h = getattr(self, "_L", None), getattr(self, "_h", None)
        if L is not None and h:
            L.gpurir_batch_destroy(h)
            self._h = None
