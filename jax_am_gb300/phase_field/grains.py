"""Grain statistics of a phase-field solution on the GPU.

The reference finds grains after a run (``jax_am/phase_field/utils.py:
181-310``, ``process_eta``): face-adjacent solid cells (T < T_liquidus) of the
same argmax orientation form a grain; grains are listed by orientation, then
in order of their smallest cell index; each grain gets its volume and the PCA
aspect ratio ``2 l0 / (l1 + l2)`` (``l`` = square roots of the explained
variances of its volume-weighted cell centres, descending), or 1 when it has
fewer than 5 cells.

``segment_grains`` runs the connected-component labelling, the per-grain
moment sums (``pfg_grains``) and the aspect ratios (one 3 x 3 eigenproblem per
grain from its exact integer moments, ``pfg_grain_shapes``) on the GPU; the host
sorts the grains.  ``process_eta`` is the drop-in for the reference function,
reading the solution that ``PFSolver.write_sols`` wrote.

A collinear grain (all cells on one line) has two zero variances: its
aspect ratio is ``inf`` here, where the reference's floating-point PCA may
return a huge finite number instead.
"""
import ctypes
import os

import numpy as np
import torch

from .. import _lib
from .allen_cahn import as_device_f32, make_pf_params


class _Box:
    """What make_pf_params reads from a polycrystal, for a grid without one."""

    def __init__(self, h, n):
        self.mesh_h_xyz = h
        self.unique_grain_directions = np.zeros((3, n, 3))


def _cell_size(pf_args):
    if all(k in pf_args for k in ("domain_x", "domain_y", "domain_z")):
        return (pf_args["domain_x"] / pf_args["Nx"], pf_args["domain_y"] / pf_args["Ny"],
                pf_args["domain_z"] / pf_args["Nz"])
    h = pf_args.get("h", 1.0)
    return tuple(h) if not np.isscalar(h) else (h, h, h)


def _cell_volume(pf_args):
    """The reference's uniform cell volume domain_vol / N (utils.py:204-205)."""
    N = int(pf_args["Nx"]) * int(pf_args["Ny"]) * int(pf_args["Nz"])
    if all(k in pf_args for k in ("domain_x", "domain_y", "domain_z")):
        return pf_args["domain_x"] * pf_args["domain_y"] * pf_args["domain_z"] / N
    hx, hy, hz = _cell_size(pf_args)
    return hx * hy * hz


_FIRST_ROWS = 4096  # grains that the first copy to the host has room for


def segment_grains(pf_args, ori_inds, T, T_ghosted=False, max_grains=None):
    """Grains of an orientation map.

    ``ori_inds``: (N,) orientation index per cell (the argmax of eta);
    ``T``: (N,) or (N, 1) per-cell temperature, or the ghosted heat state with
    ``T_ghosted``.  Returns a dict with ``labels`` ((N,) int32 CUDA tensor,
    grain number in the reference's order, -1 in liquid), ``ori``,
    ``first_cell``, ``cells``, ``volumes`` and ``aspect_ratios`` (NumPy, one
    entry per grain in the reference's order)."""
    lib = _lib.load()
    N = int(pf_args["Nx"]) * int(pf_args["Ny"]) * int(pf_args["Nz"])
    ori = torch.as_tensor(np.asarray(ori_inds) if not torch.is_tensor(ori_inds) else ori_inds)
    ori = ori.to("cuda", torch.int32).reshape(-1).contiguous()
    if ori.numel() != N:
        raise ValueError(f"ori_inds has {ori.numel()} entries, expected {N}")
    n = int(pf_args.get("num_oris", 0))
    if n < 1:  # not given: from the map
        n = max(n, int(ori.max().item()) + 1 if N else 1)
    args = dict(pf_args, num_oris=min(n, _lib.MAX_ORIS))
    for key, default in (("gas_const", 8.3), ("Qg", 1.4e5), ("L0", 3.5e3), ("kappa_g", 2.77e-6),
                         ("m_g", 2.4e5), ("anisotropy", 0.0), ("ad_hoc", 1.0)):
        args.setdefault(key, default)
    params = make_pf_params(args, _Box(_cell_size(pf_args), args["num_oris"]))
    T = as_device_f32(T, None, "T").reshape(-1)
    expect = (N if not T_ghosted else
              (int(pf_args["Nx"]) + 2) * (int(pf_args["Ny"]) + 2) * (int(pf_args["Nz"]) + 2))
    if T.numel() != expect:
        raise ValueError(f"T has {T.numel()} entries, expected {expect}")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nbytes = int(lib.pfg_grain_scratch_bytes(ctypes.byref(params)))
    scratch = torch.empty(max(nbytes, 16), dtype=torch.uint8, device="cuda")
    labels = torch.empty(N, dtype=torch.int32, device="cuda")
    rec = ctypes.sizeof(_lib.Grain) // 8
    cap = int(max_grains) if max_grains else max(1024, N // 64)
    while True:
        buf = torch.empty(max(cap, 1) * rec, dtype=torch.int64, device="cuda")
        # the count, then a row of four words per grain: one copy brings both
        shapes = torch.empty((cap + 1, 4), dtype=torch.int64, device="cuda")
        st = lib.pfg_grains(ctypes.byref(params), _lib.ptr(ori), _lib.ptr(T), int(T_ghosted),
                            _lib.ptr(labels), _lib.ptr(buf), cap, _lib.ptr(shapes),
                            _lib.ptr(scratch), scratch.numel(), stream)
        _lib.check(st, "pfg_grains")
        st = lib.pfg_grain_shapes(_lib.ptr(buf), _lib.ptr(shapes), cap,
                                  ctypes.c_void_p(shapes.data_ptr() + 32), stream)
        _lib.check(st, "pfg_grain_shapes")
        host = shapes[: min(cap, _FIRST_ROWS) + 1].cpu()
        K = int(host[0, 0])
        if K <= cap:
            break
        cap = K
    if K >= len(host):
        host = shapes[: K + 1].cpu()
    raw = host[1: K + 1].numpy()
    # column 1 holds (ori, reserved) as two little-endian int32
    ori_g = raw[:, 1] & 0xFFFFFFFF
    # by orientation, then smallest cell index (the order of the rows)
    order = np.argsort(ori_g, kind="stable")
    if K:
        rank = np.empty(K, dtype=np.int32)
        rank[order] = np.arange(K, dtype=np.int32)
        rank_t = torch.from_numpy(rank).to("cuda")
        st = lib.pfg_grain_relabel(N, _lib.ptr(rank_t), _lib.ptr(labels), stream)
        _lib.check(st, "pfg_grain_relabel")
    raw = raw[order]
    cells = np.ascontiguousarray(raw[:, 2])
    return {
        "labels": labels,
        "ori": ori_g[order],
        "first_cell": np.ascontiguousarray(raw[:, 0]),
        "cells": cells,
        "volumes": cells * _cell_volume(pf_args),
        "aspect_ratios": np.ascontiguousarray(raw[:, 3]).view(np.float64),
    }


def process_eta(pf_args, step=13):
    """Drop-in for the reference's ``process_eta`` (utils.py:181-214): reads
    the solution ``PFSolver.write_sols`` wrote for ``step`` (``<data_dir>/
    numpy/pf/sols/u<step>.npz``; the reference reads the VTU it wrote) and
    returns ``[grain volumes, grain aspect ratios]`` in the reference's grain
    order."""
    path = os.path.join(pf_args["data_dir"], f"numpy/pf/sols/u{step:03d}.npz")
    d = np.load(path)
    res = segment_grains(pf_args, d["ori_inds"], d["T"])
    return [list(res["volumes"]), list(res["aspect_ratios"])]
