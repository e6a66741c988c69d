"""Accessibility on the GPU (DataMap.accessibility with angular = False, rust/src/data.rs:605-740):
the data map's tables go to the device once per call and cs_accessibility runs one search per live
source, summing its reachable entries per land-use class and threshold."""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _native, centrality


def accessibility_rows(ns, t: dict, sources, d, b, s, mcw, speed: float, n_classes: int):
    """Per class: unweighted and weighted rows [n_classes][K][n_bound] (f64) and the nearest
    distance within the largest threshold [n_classes][n_bound] (NaN when none), for `sources`."""
    nb = ns.node_bound()
    K = len(d)
    if n_classes == 0 or len(sources) == 0:
        return np.zeros((n_classes, K, nb)), np.zeros((n_classes, K, nb)), np.full((n_classes, nb), np.nan)
    csr = centrality._primal_csr(ns)
    dev = csr.device
    ws = centrality._workspace(ns, csr, 0, 1, speed, int(max(s)))

    i32 = ("ptr", "a_entry", "a_node", "a_rank", "entry_group", "entry_class", "g_ptr", "g_assign")
    names = ("node_ptr", "assign_entry", "assign_node", "assign_rank", "entry_group", "entry_class", "group_ptr",
             "group_assign")
    # every table, the sources and the (unused) source weights and eligibility in one copy
    *tables, dist_t, src_t, zf, zu = centrality.upload(
        [np.asarray(t[k], np.int32) for k in i32] + [np.asarray(t["a_dist"], np.float32), np.asarray(sources, np.int32),
                                                     np.zeros(1, np.float32), np.zeros(1, np.uint8)], dev)
    keep = dict(zip(names, tables), assign_dist=dist_t)
    dm = _native.DataMapArrays()
    dm.n_entries = len(t["keys"])
    dm.n_assign = len(t["a_entry"])
    dm.n_groups = int(t["n_groups"])
    for name, tensor in keep.items():
        setattr(dm, name, tensor.data_ptr() if tensor.numel() else None)
    q = centrality._make_query(d, b, s, speed, float(centrality.TIE_EPSILON), False, False, False, src_t, zf, zu)
    # both f64 rows, then the f32 nearest distances, in one buffer
    m = n_classes * K * nb
    buf = torch.zeros(2 * m + (n_classes * nb + 1) // 2, dtype=torch.float64, device=dev)
    unw, wt, near = buf[:m], buf[m:2 * m], buf[2 * m:].view(torch.float32)
    near.fill_(float("inf"))
    mcw_arr = (C.c_float * K)(*[float(x) for x in mcw])
    lib = _native.load()
    rc = lib.cs_accessibility(C.byref(csr.struct(speed)), C.byref(dm), C.byref(q), mcw_arr, int(n_classes),
                              C.byref(ws.plan), ws.ptr, ws.nbytes, unw.data_ptr(), wt.data_ptr(), near.data_ptr(),
                              centrality._stream_ptr())
    if rc != _native.CS_OK:
        ws.init(centrality._stream_ptr())
    _native.check(rc, "cs_accessibility")
    host = buf.cpu().numpy()
    near_h = host[2 * m:].view(np.float32)[:n_classes * nb].reshape(n_classes, nb).astype(np.float64)
    near_h[np.isinf(near_h)] = np.nan
    return host[:m].reshape(n_classes, K, nb), host[m:2 * m].reshape(n_classes, K, nb), near_h
