"""Host prepare: tree topology and interaction lists (yggdrax stand-in).

``build_topology`` calls ``jb_tree_build`` (csrc/tree_build.cpp) and returns a
:class:`Topology` of numpy arrays in the layout the reference's kernels read
from yggdrax artefacts (``Tree.node_ranges/left_child/right_child``,
``NodeInteractionList``, ``NodeNeighborList``, the Morton permutation), see
jaccpot/runtime/fmm_state.py:870-897 for the state that carries them.
"""

from __future__ import annotations

import ctypes
from dataclasses import dataclass, field, fields

import numpy as np

from . import _lib


@dataclass
class Topology:
    num_particles: int
    num_nodes: int
    num_internal: int
    num_leaves: int
    num_levels: int
    max_leaf_occupancy: int
    leaf_size: int
    theta: float
    permutation: np.ndarray  # int64[N] sorted slot -> input index
    inverse_permutation: np.ndarray  # int64[N] input index -> sorted slot
    node_ranges: np.ndarray  # int32[num_nodes, 2] inclusive
    left_child: np.ndarray  # int32[num_internal]
    right_child: np.ndarray  # int32[num_internal]
    parent: np.ndarray  # int32[num_nodes]
    node_level: np.ndarray  # int32[num_nodes]
    level_offsets: np.ndarray  # int32[num_levels + 1]
    leaf_of_particle: np.ndarray  # int32[N]
    far_offsets: np.ndarray  # int64[num_nodes + 1]
    far_sources: np.ndarray  # int32[num_far]
    near_offsets: np.ndarray  # int64[num_leaves + 1]
    near_leaves: np.ndarray  # int32[num_near]
    centers_f64: np.ndarray  # float64[num_nodes, 3] (host COM used by the MAC)
    radii_f64: np.ndarray  # float64[num_nodes]
    m2l_targets: np.ndarray = field(default=None)  # int32, nodes with >= 1 far pair, longest list first
    # error-controlled walk only: gear index of every far pair and the gears' orders
    far_gears: np.ndarray = field(default=None)  # int32[num_far]
    gear_orders: tuple = field(default=None)

    @property
    def num_far_pairs(self) -> int:
        return int(self.far_sources.shape[0])

    @property
    def num_near_pairs(self) -> int:
        return int(self.near_leaves.shape[0])

    def far_pair_targets(self) -> np.ndarray:
        """int32[num_far]: the target node of every far pair (CSR row of each entry)."""
        return np.repeat(np.arange(self.num_nodes, dtype=np.int32), np.diff(self.far_offsets)).astype(np.int32)

    def far_reverse_index(self) -> np.ndarray:
        """int32[num_far]: index of the pair (s <- t) for every pair (t <- s).

        The dual traversal emits every accepted pair in both directions, so the
        reverse always exists; raises if it does not (the adjoint relies on it)."""
        tgt = self.far_pair_targets().astype(np.int64)
        src = self.far_sources.astype(np.int64)
        key = tgt * self.num_nodes + src
        order = np.argsort(key, kind="stable")
        rkey = src * self.num_nodes + tgt
        pos = np.searchsorted(key[order], rkey)
        pos = np.minimum(pos, max(key.size - 1, 0))
        rev = order[pos] if key.size else np.zeros(0, np.int64)
        if key.size and not np.array_equal(key[rev], rkey):
            raise ValueError("far lists are not symmetric")
        return rev.astype(np.int32)

    def near_lists_symmetric(self) -> bool:
        """True when leaf B is in A's neighbour list exactly when A is in B's."""
        tgt = np.repeat(np.arange(self.num_leaves, dtype=np.int64), np.diff(self.near_offsets))
        src = self.near_leaves.astype(np.int64)
        a = np.sort(tgt * self.num_leaves + src)
        b = np.sort(src * self.num_leaves + tgt)
        return bool(np.array_equal(a, b))

    def near_pair_interactions(self) -> int:
        """Particle-particle interactions of the near field (self blocks included)."""
        cnt = (self.node_ranges[:, 1] - self.node_ranges[:, 0] + 1).astype(np.int64)
        leaf_cnt = cnt[self.num_internal:]
        src_cnt = leaf_cnt[self.near_leaves]
        per_edge_t = np.repeat(leaf_cnt, np.diff(self.near_offsets))
        return int((per_edge_t * src_cnt).sum() + (leaf_cnt * (leaf_cnt - 1)).sum())


class _OnFirstRead:
    """A DeviceBuiltTopology field that Topology gives a default: the instance's
    own value, else the one brought from the device."""

    def __set_name__(self, owner, name):
        self.name = name

    def __get__(self, obj, owner=None):
        return None if obj is None else obj._host(self.name)

    def __set__(self, obj, value):
        obj.__dict__[self.name] = value


class DeviceBuiltTopology(Topology):
    """A Topology whose arrays are on the GPU (``device_arrays``, torch tensors
    that own their memory) and come to the host one by one, when they are first
    read as numpy arrays; from then on the host's array is the field.  An
    evaluation needs only the sizes and the level offsets there: at clustered
    1M the copies down and up again were 35 of the 52 ms that the GPU was busy
    in a call on new particles, and most of the host's 140 ms.

    The tensors are filled in order on the stream that was current when the
    object was made; reads on the host, and ``device_array`` under another
    stream, wait for that."""

    m2l_targets = _OnFirstRead()
    far_gears = _OnFirstRead()
    gear_orders = None

    @staticmethod
    def of(n: int, info, arrays: dict, level_offsets: np.ndarray, leaf_size: int, theta: float,
           gear_orders=None) -> "DeviceBuiltTopology":
        t = object.__new__(DeviceBuiltTopology)
        t.num_particles = n
        for name in ("num_nodes", "num_internal", "num_leaves", "num_levels", "max_leaf_occupancy"):
            setattr(t, name, int(getattr(info, name)))
        t.leaf_size, t.theta = int(leaf_size), float(theta)
        t.level_offsets = level_offsets
        t.gear_orders = None if gear_orders is None else tuple(int(o) for o in gear_orders)
        t._sizes = _field_sizes(n, info)
        t._take(arrays, {})
        return t

    def _take(self, arrays: dict, streams: dict) -> None:
        """The tensors, those without an entry in `streams` (the stream they
        belong to) being of the current one, and an event behind what fills them."""
        import torch

        device = next(iter(arrays.values())).device
        here = _lib.stream_handle(device)
        self.device_arrays = arrays
        self._streams = {name: streams.get(name, here) for name in arrays}
        self._ready = torch.cuda.Event()
        self._ready.record(torch.cuda.current_stream(device))

    @property
    def num_far_pairs(self) -> int:
        return int(self.far_sources.shape[0]) if "far_sources" in self.__dict__ else self._sizes["far_sources"]

    @property
    def num_near_pairs(self) -> int:
        return int(self.near_leaves.shape[0]) if "near_leaves" in self.__dict__ else self._sizes["near_leaves"]

    def device_array(self, name: str, stream: int | None = None):
        """The field's tensor, with at least one element, for use on the current
        stream (`stream`: its handle, for callers that have it); None when the
        field has been read on the host, whose array then counts."""
        a = None if name in self.__dict__ else self.__dict__.get("device_arrays", {}).get(name)
        if a is not None and (_lib.stream_handle(a.device) if stream is None else stream) != self._streams[name]:
            import torch

            here = torch.cuda.current_stream(a.device)
            here.wait_event(self._ready)
            a.record_stream(here)  # its memory waits for this use before it serves another
        return a

    def with_geometry(self, centers_f64, radii_f64) -> "DeviceBuiltTopology":
        """The same tree and lists with other centres and radii (device tensors
        of the current stream)."""
        import torch

        t = object.__new__(DeviceBuiltTopology)
        t.__dict__.update(self.__dict__)
        moved = {"centers_f64": centers_f64, "radii_f64": radii_f64}
        for name in moved:
            t.__dict__.pop(name, None)
        torch.cuda.current_stream(centers_f64.device).wait_event(self._ready)  # one event for both
        t._take({**self.device_arrays, **moved}, {k: s for k, s in self._streams.items() if k not in moved})
        return t

    def __reduce__(self):
        """Copies and saved files are plain Topologies of host arrays, which a
        process without a GPU can load."""
        return Topology, tuple(getattr(self, f.name) for f in fields(Topology))

    def _host(self, name: str):
        d = self.__dict__
        if name not in d:
            if name == "m2l_targets":
                d[name] = _m2l_targets(self.far_offsets)
            elif name not in d.get("device_arrays", {}):  # far_gears without an error-controlled walk
                return None
            else:
                self._ready.synchronize()
                a = d["device_arrays"][name][:self._sizes[name]].cpu().numpy()
                d[name] = a.reshape({"node_ranges": (-1, 2), "centers_f64": (-1, 3)}.get(name, (-1,)))
        return d[name]

    def __getattr__(self, name: str):  # a field that the instance does not hold yet
        if name in _LAZY_FIELDS and "device_arrays" in self.__dict__:
            return self._host(name)
        raise AttributeError(name)


_LAZY_FIELDS = frozenset(_lib.DTREE_FIELDS) - {"level_offsets", "far_gears"}


def _field_sizes(n: int, info) -> dict:
    return {
        "permutation": n,
        "inverse_permutation": n,
        "node_ranges": 2 * info.num_nodes,
        "left_child": info.num_internal,
        "right_child": info.num_internal,
        "parent": info.num_nodes,
        "node_level": info.num_nodes,
        "level_offsets": info.num_levels + 1,
        "leaf_of_particle": n,
        "far_offsets": info.num_nodes + 1,
        "far_sources": info.num_far_pairs,
        "near_offsets": info.num_leaves + 1,
        "near_leaves": info.num_near_pairs,
        "centers_f64": 3 * info.num_nodes,
        "radii_f64": info.num_nodes,
        "far_gears": info.num_far_pairs,
    }


def _copy_fields(copy_fn, handle, n: int, info) -> dict:
    sizes = _field_sizes(n, info)
    arrs = {}
    for name, (fid, dt) in _lib.TREE_FIELDS.items():
        if name == "far_gears":  # error-controlled walks run on the GPU only
            continue
        a = np.empty(max(sizes[name], 1), dtype=dt)
        _lib.check(copy_fn(handle, fid, a.ctypes.data), f"tree field copy ({name})")
        arrs[name] = a[: sizes[name]]
    return arrs


def _m2l_targets(far_offsets: np.ndarray) -> np.ndarray:
    """int32: the nodes with at least one far pair, longest list first (stable)."""
    counts = np.diff(far_offsets)
    tg = np.nonzero(counts)[0]
    return tg[np.argsort(-counts[tg], kind="stable")].astype(np.int32)


def _topology(n: int, info, arrs: dict, leaf_size: int, theta: float) -> Topology:
    perm = arrs["permutation"]
    inv = np.empty_like(perm)
    inv[perm] = np.arange(n, dtype=np.int64)
    return Topology(
        num_particles=n,
        num_nodes=info.num_nodes,
        num_internal=info.num_internal,
        num_leaves=info.num_leaves,
        num_levels=info.num_levels,
        max_leaf_occupancy=info.max_leaf_occupancy,
        leaf_size=int(leaf_size),
        theta=float(theta),
        permutation=perm,
        inverse_permutation=inv,
        node_ranges=arrs["node_ranges"].reshape(-1, 2),
        left_child=arrs["left_child"],
        right_child=arrs["right_child"],
        parent=arrs["parent"],
        node_level=arrs["node_level"],
        level_offsets=arrs["level_offsets"],
        leaf_of_particle=arrs["leaf_of_particle"],
        far_offsets=arrs["far_offsets"],
        far_sources=arrs["far_sources"],
        near_offsets=arrs["near_offsets"],
        near_leaves=arrs["near_leaves"],
        centers_f64=arrs["centers_f64"].reshape(-1, 3),
        radii_f64=arrs["radii_f64"],
        m2l_targets=_m2l_targets(arrs["far_offsets"]),
    )


def build_topology(positions, masses, *, leaf_size: int = 16, theta: float = 0.6, device=None) -> Topology:
    """Tree + lists on the host (``jb_tree_build``), or on the GPU
    (``jb_tree_build_device``, the same arrays bit for bit) when ``device`` is
    a CUDA device."""
    if device is not None and str(device).startswith("cuda"):
        return build_topology_device(positions, masses, leaf_size=leaf_size, theta=theta, device=device)
    host = lambda a: a.detach().cpu().numpy() if hasattr(a, "detach") else a
    pos = np.ascontiguousarray(np.asarray(host(positions), dtype=np.float64).reshape(-1, 3))
    mass = np.ascontiguousarray(np.asarray(host(masses), dtype=np.float64).reshape(-1))
    n = pos.shape[0]
    if mass.shape[0] != n:
        raise ValueError("positions and masses disagree in length")
    lb = _lib.lib()
    h = ctypes.c_void_p()
    _lib.check(lb.jb_tree_build(n, pos.ctypes.data, mass.ctypes.data, int(leaf_size), float(theta),
                                ctypes.byref(h)), "jb_tree_build")
    try:
        info = _lib.TreeInfo()
        _lib.check(lb.jb_tree_info(h, ctypes.byref(info)), "jb_tree_info")
        arrs = _copy_fields(lb.jb_tree_copy, h, n, info)
    finally:
        lb.jb_tree_free(h)
    return _topology(n, info, arrs, leaf_size, theta)


def _torch_dtype(dtype):
    import torch

    return {"i4": torch.int32, "i8": torch.int64, "f8": torch.float64}[dtype.str[1:]]


class _View:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def device_view(ptr, shape, dtype, device):
    """Zero-copy torch view (``__cuda_array_interface__`` v3) of device memory
    owned by a library handle; valid while the handle lives."""
    import torch

    dtype = np.dtype(dtype)
    shape = tuple(int(x) for x in shape)
    if int(np.prod(shape)) == 0:
        return torch.zeros(shape, dtype=torch.from_numpy(np.zeros(0, dtype)).dtype, device=device)

    return torch.as_tensor(_View(ptr, shape, dtype.str), device=device)


class DeviceTree:
    """Owner of a ``jb_tree_build_device`` handle: the tree and lists of a
    particle set, resident on the GPU.  ``field(name)`` is a zero-copy torch
    view of one array (valid while the handle lives); ``topology()`` copies
    everything into tensors of its own, as a :class:`DeviceBuiltTopology`.
    Use as a context manager or call ``free()``."""

    def __init__(self, positions, masses, *, leaf_size: int = 16, theta: float = 0.6, device="cuda"):
        import torch

        self._torch = torch
        pos = torch.as_tensor(positions).to(device=device, dtype=torch.float64).reshape(-1, 3).contiguous()
        mass = torch.as_tensor(masses).to(device=device, dtype=torch.float64).reshape(-1).contiguous()
        n = pos.shape[0]
        if mass.shape[0] != n:
            raise ValueError("positions and masses disagree in length")
        self.n, self.leaf_size, self.theta, self.device = int(n), int(leaf_size), float(theta), pos.device
        self._lb = _lib.lib()
        self._h = ctypes.c_void_p()
        stream = _lib.stream_handle(pos.device)
        self._streams = {stream}  # the handle's buffers are freed on these
        _lib.check(self._lb.jb_tree_build_device(n, pos.data_ptr(), mass.data_ptr(), self.leaf_size, self.theta,
                                                 stream, ctypes.byref(self._h)), "jb_tree_build_device")
        self.info = _lib.TreeInfo()
        _lib.check(self._lb.jb_dtree_info(self._h, ctypes.byref(self.info)), "jb_dtree_info")
        self.sizes = _field_sizes(self.n, self.info)
        self.gear_orders = None  # set by adaptive_walk

    def adaptive_walk(self, power, force_scale, *, G: float, eps: float, theta_max: float = 1.0,
                      gear_orders=(8,)) -> None:
        """Replaces the lists by those of the error-controlled walk
        (jb_dtree_adaptive_walk: Dehnen eq. (15)/(16a) acceptance, target-
        centric, per-pair gears).  power: float64 (num_nodes, P+1) Dehnen
        source powers; force_scale: float32 (num_nodes,) -- both on this
        tree's device, in its node order."""
        torch = self._torch
        orders = np.ascontiguousarray(np.asarray(gear_orders, dtype=np.int32))
        pw = power.to(device=self.device, dtype=torch.float64).contiguous()
        fs = force_scale.to(device=self.device, dtype=torch.float32).contiguous()
        if pw.dim() != 2 or pw.shape[0] != self.info.num_nodes or fs.shape != (self.info.num_nodes,):
            raise ValueError("power must be (num_nodes, P+1) and force_scale (num_nodes,)")
        stream = _lib.stream_handle(self.device)
        self._streams.add(stream)
        _lib.check(self._lb.jb_dtree_adaptive_walk(self._h, int(pw.shape[1]), pw.data_ptr(), fs.data_ptr(),
                                                   float(G), float(eps), float(theta_max), int(orders.size),
                                                   orders.ctypes.data, stream), "jb_dtree_adaptive_walk")
        _lib.check(self._lb.jb_dtree_info(self._h, ctypes.byref(self.info)), "jb_dtree_info")
        self.sizes = _field_sizes(self.n, self.info)
        self.gear_orders = tuple(int(o) for o in orders)

    def field(self, name: str):
        fid, dt = _lib.DTREE_FIELDS[name]
        return device_view(self._lb.jb_dtree_field(self._h, fid), (self.sizes[name],), dt, self.device)

    def topology(self) -> DeviceBuiltTopology:
        """Tree and lists in one device buffer that the topology owns (copied
        in stream order, one call); only the level offsets come to the host."""
        torch = self._torch
        names = [f for f in _lib.DTREE_FIELDS if f != "far_gears" or self.gear_orders is not None]
        at, spans = 0, {}
        for f in names:
            dtype = np.dtype(_lib.DTREE_FIELDS[f][1])
            count = max(self.sizes[f], 1)  # an empty field keeps a word, so that its pointer is never null
            spans[f] = (at, count, dtype)
            at += (count * dtype.itemsize + 255) & ~255
        buf = torch.empty(at, dtype=torch.uint8, device=self.device)
        base = buf.data_ptr()
        ids = np.array([_lib.DTREE_FIELDS[f][0] for f in names], dtype=np.int32)
        dst = np.array([base + spans[f][0] for f in names], dtype=np.uint64)
        stream = _lib.stream_handle(self.device)
        _lib.check(self._lb.jb_dtree_export(self._h, len(names), ids.ctypes.data, dst.ctypes.data, stream),
                   "jb_dtree_export")
        arrays = {f: buf[o:o + c * d.itemsize].view(_torch_dtype(d)) for f, (o, c, d) in spans.items()}
        for f in names:
            if self.sizes[f] == 0:
                arrays[f].zero_()
        for s in self._streams - {stream}:  # the copies are done before a buffer is freed
            _lib.check(self._lb.jb_stream_wait(s, stream), "jb_stream_wait")
        offsets = np.empty(self.info.num_levels + 1, dtype=np.int32)
        _lib.check(self._lb.jb_dtree_copy(self._h, _lib.DTREE_FIELDS["level_offsets"][0], offsets.ctypes.data),
                   "tree field copy (level_offsets)")
        return DeviceBuiltTopology.of(self.n, self.info, arrays, offsets, self.leaf_size, self.theta,
                                      self.gear_orders)

    def free(self) -> None:
        if self._h:
            self._lb.jb_dtree_free(self._h)
            self._h = ctypes.c_void_p()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.free()

    def __del__(self):
        try:
            self.free()
        except Exception:  # interpreter shutdown
            pass


def build_topology_device(positions, masses, *, leaf_size: int = 16, theta: float = 0.6, device="cuda") -> Topology:
    """The tree and lists built on the GPU by ``jb_tree_build_device``
    (csrc/tree_gpu.cu) from float64 copies of the inputs on ``device``: the
    host build's :class:`Topology`, its arrays copied to the host when read."""
    with DeviceTree(positions, masses, leaf_size=leaf_size, theta=theta, device=device) as dtree:
        return dtree.topology()
