"""ctypes binding of ``libdwba_b200.so`` (the C ABI in ``include/dwba_b200.h``).

The shared library is built in-tree by ``dwba_b200/build.py``. Loading fails
loudly: there is no CPU fallback for the engine.
"""
from __future__ import annotations

import ctypes
import os

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "libdwba_b200.so")

DWBA_OK = 0
DWBA_ERR_INVALID_ARG = 1
DWBA_ERR_CUDA = 2
DWBA_ERR_NO_DEVICE = 3
DWBA_ERR_WORKSPACE = 4
DWBA_ERR_UNSUPPORTED = 5
DWBA_ERR_RANGE = 6
DWBA_MAX_L = 63

# Struct layouts (must match include/dwba_b200.h; checked against the library at load).
NODESET_DTYPE = np.dtype([(n, "<u8") for n in ("r", "logr", "breaks", "ta", "bx")]
                         + [(n, "<i4") for n in ("n_grid", "n1", "n_breaks", "log1", "log2", "pad")])
FOLD_DTYPE = np.dtype([(n, "<u8") for n in ("op", "f", "g", "out")]
                      + [(n, "<i4") for n in ("half_band", "n_out", "n_src", "n_clear")])
FORM_DTYPE = np.dtype([("r", "<u8"), ("a", "<u8"), ("b", "<u8"), ("n_rows", "<i4"), ("n_cols", "<i4")])
FORM_GRAD_DTYPE = np.dtype([("r", "<u8"), ("a", "<u8"), ("b", "<u8"), ("ga", "<u8"), ("gb", "<u8"),
                            ("n_rows", "<i4"), ("n_cols", "<i4")])
FOLD_ADJ_DTYPE = np.dtype([("op", "<u8"), ("y", "<u8"), ("z", "<u8"), ("half_band", "<i4"), ("n_out", "<i4"),
                           ("n_src", "<i4"), ("pad", "<i4")])
FOLD_MULTI = 8
FOLD_MULTI_DTYPE = np.dtype([("op", "<u8"), ("g", "<u8"), ("f", "<u8", (FOLD_MULTI,)), ("out", "<u8", (FOLD_MULTI,)),
                             ("n_f", "<i4"), ("half_band", "<i4"), ("n_out", "<i4"), ("n_src", "<i4"),
                             ("n_clear", "<i4"), ("pad", "<i4")])
POTENTIAL_DTYPE = np.dtype([("r", "<u8"), ("b", "<u8"), ("phi", "<u8"), ("n_rows", "<i4"), ("n_cols", "<i4"),
                            ("stride", "<i4"), ("pad", "<i4")])
DOT_DTYPE = np.dtype([("a", "<u8"), ("phi", "<u8"), ("out", "<u8"), ("n_rows", "<i4"), ("stride", "<i4")])
DENSE_RUN = 8  # descriptors per run sharing a grid (dwba_dense_potentials)
DOT_RUN = 16  # descriptors per run sharing one potential (dwba_dot_forms)
CUPY_SET_DTYPE = np.dtype([("r", "<u8"), ("logr", "<u8"), ("ops", "<u8"), ("n1", "<i4"), ("n_breaks", "<i4"),
                           ("L_max", "<i4"), ("pad", "<i4")])
CUPY_FORM_DTYPE = np.dtype([("r", "<u8"), ("a", "<u8"), ("f", "<u8"), ("g", "<u8"), ("ops", "<u8"), ("out", "<u8"),
                            ("n1", "<i4"), ("L_max", "<i4")])
TC_SEGMENT_DTYPE = np.dtype([("forms", "<u8"), ("r", "<u8"), ("out", "<u8"), ("n_forms", "<i4"), ("n_grid", "<i4")])
TC_TILE_DTYPE = np.dtype([("bn", "<i4"), ("stages", "<i4"), ("order", "<i4"), ("pad", "<i4")])
PANEL_COL_DTYPE = np.dtype([("phi", "<u8"), ("mul", "<u8")])
PANEL_DTYPE = np.dtype([("rows", "<u8"), ("cols", "<u8"), ("out", "<u8"), ("part_off", "<i8"), ("M", "<i4"), ("F", "<i4"),
                        ("n", "<i4"), ("stride", "<i4")])
PANEL_CTA_DTYPE = np.dtype([("panel", "<i4"), ("m_tile", "<i4"), ("n_tile", "<i4"), ("chunk", "<i4")])
PANEL_ENTRY_DTYPE = np.dtype([(n, "<i4") for n in ("set", "t", "w_i", "w_f", "u_i", "u_f")])
PANEL_LAYOUT_ARRAYS = ("ia", "ib", "a_u", "a_w", "a_set", "b_u", "b_w", "b_set", "psi_t", "psi_set", "d_M", "d_F", "d_set",
                       "d_rows", "d_psi", "d_wave", "d_entry", "x_M", "x_F", "x_set", "x_rows", "x_cols", "x_entry")
PANEL_LAYOUT_DTYPE = np.dtype([(n, "<u8") for n in PANEL_LAYOUT_ARRAYS]
                              + [(n, "<i4") for n in ("n_a", "n_b", "n_psi", "n_direct", "n_exchange", "pad")])
TAIL_DTYPE = np.dtype([("wave", "<f8", (10,)), ("r_m", "<f8"), ("r_max", "<f8"), ("moments", "<u8"), ("out", "<u8"),
                       ("mode", "<i4"), ("pad", "<i4")])


class DWBAError(RuntimeError):
    """Non-zero status from the C ABI."""

    def __init__(self, status: int, where: str):
        self.status = status
        super().__init__(f"{where}: {status_string(status)} (status {status})")


_lib = None


def _declare(lib):
    c_int, c_i64, c_dbl, c_vp = ctypes.c_int, ctypes.c_int64, ctypes.c_double, ctypes.c_void_p
    sig = {
        "dwba_abi_version": (c_int, []),
        "dwba_status_string": (ctypes.c_char_p, [c_int]),
        "dwba_device_probe": (c_int, [ctypes.POINTER(c_int)] * 3),
        "dwba_struct_sizes": (c_int, [ctypes.POINTER(c_i64), c_int]),
        "dwba_build_nodesets": (c_int, [c_vp, c_int, c_int, c_vp, c_vp, c_int, c_vp, c_vp]),
        "dwba_build_nodesets_folded": (c_int, [c_vp, c_vp, c_int, c_int, c_vp, c_vp, c_int, c_vp, c_vp]),
        "dwba_fold": (c_int, [c_vp, c_int, c_int, c_vp]),
        "dwba_dense_chunk_prefix": (c_i64, [c_vp, c_int, c_vp]),
        "dwba_bilinear_dense_fp64": (c_int, [c_vp, c_int, c_int, c_vp, c_vp, c_i64, c_vp, c_i64, c_vp, c_vp]),
        "dwba_bilinear_semisep_fp64": (c_int, [c_vp, c_int, c_int, c_vp, c_dbl, c_dbl, c_vp, c_vp]),
        "dwba_bilinear_semisep_abs_fp64": (c_int, [c_vp, c_int, c_int, c_vp, c_dbl, c_dbl, c_vp, c_vp]),
        "dwba_bilinear_dense_fp64_noalloc": (c_int, [c_vp, c_int, c_int, c_int, c_vp, c_vp, c_vp]),
        "dwba_tc_workspace_bytes": (c_i64, [c_int, c_int, c_int, c_int]),
        "dwba_bilinear_tc_bf16": (c_int, [c_vp, c_int, c_vp, c_int, c_int, c_int, c_vp, c_vp, c_i64, c_vp, c_vp,
                                          c_vp]),
        "dwba_phase_breaks_coulomb": (c_int, [c_dbl, c_dbl, c_dbl, c_dbl, c_dbl, c_vp, c_int,
                                              ctypes.POINTER(c_int)]),
        "dwba_outer_tails": (c_int, [c_vp, c_dbl, c_dbl, c_int, c_vp, c_int, c_int, c_dbl, c_vp]),
        "dwba_outer_tails_batch": (c_int, [c_vp, c_int, c_int, c_int, c_dbl, c_vp]),
        "dwba_bilinear_semisep_backward_fp64": (c_int, [c_vp, c_int, c_int, c_vp, c_vp, c_dbl, c_dbl, c_vp]),
        "dwba_fold_adjoint": (c_int, [c_vp, c_int, c_int, c_vp]),
        "dwba_tc_backward_workspace_bytes": (c_i64, [c_int, c_int, c_int, c_int]),
        "dwba_bilinear_tc_bf16_backward": (c_int, [c_vp, c_int, c_vp, c_int, c_int, c_int, c_vp, c_vp, c_vp, c_i64,
                                                   c_vp, c_vp]),
        "dwba_fold_multi": (c_int, [c_vp, c_int, c_int, c_vp]),
        "dwba_cross_sections": (c_int, [c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_int, c_int, c_int, c_int, c_dbl,
                                        c_vp, c_vp, c_vp]),
        "dwba_outer_tail_on_device": (c_int, [c_vp, c_dbl, c_dbl]),
        "dwba_outer_tails_on_device": (c_int, [c_vp, c_vp, c_int, c_dbl, c_vp]),
        "dwba_l0_corrections": (c_int, [c_vp, c_vp, c_vp, c_int, c_int, c_vp, c_vp, c_vp, c_vp, c_dbl, c_vp, c_vp]),
        "dwba_tc_set_wait_cycles": (c_int, [c_i64]),
        "dwba_multipole_potentials": (c_int, [c_vp, c_int, c_int, c_vp, c_dbl, c_dbl, c_vp]),
        "dwba_multipole_potentials_sized": (c_int, [c_vp, c_int, c_int, c_int, c_vp, c_dbl, c_dbl, c_vp]),
        "dwba_tc_potentials_layout": (c_i64, [c_int, c_int, c_int, c_int, ctypes.POINTER(c_i64), ctypes.POINTER(c_i64)]),
        "dwba_tc_potentials": (c_int, [c_vp, c_int, c_vp, c_int, c_int, c_int, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp]),
        "dwba_dense_potentials": (c_int, [c_vp, c_int, c_int, c_int, c_vp, c_vp]),
        "dwba_dot_forms": (c_int, [c_vp, c_int, c_int, c_vp]),
        "dwba_cupy_exchange_ops": (c_int, [c_vp, c_int, c_int, c_int, c_vp, c_vp, c_int, c_vp]),
        "dwba_cupy_exchange_forms": (c_int, [c_vp, c_int, c_int, c_dbl, c_dbl, c_vp]),
        "dwba_tc_ragged_workspace_bytes": (c_i64, [c_vp, c_int, c_int, c_int, c_vp]),
        "dwba_bilinear_tc_bf16_ragged": (c_int, [c_vp, c_int, c_int, c_int, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp]),
        "dwba_panel_layout": (c_int, [c_vp, c_int, c_int, c_int, c_int, c_dbl, c_int, c_vp]),
        "dwba_panel_plan": (c_i64, [c_vp, c_int, c_int, c_vp, ctypes.POINTER(c_i64)]),
        "dwba_panel_forms": (c_int, [c_vp, c_int, c_vp, c_i64, c_int, c_int, c_vp, c_vp]),
        "dwba_copy_from_host": (c_int, [c_vp, c_vp, c_i64, c_vp]),
    }
    for name, (res, args) in sig.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    return lib


def load():
    """Load the library (once). Raises if it is missing or its ABI does not match."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise ImportError(f"{LIB_PATH} is missing: build it with `python -m dwba_b200.build` "
                          "(the engine has no CPU fallback)")
    lib = _declare(ctypes.CDLL(LIB_PATH))
    if lib.dwba_abi_version() != 1:
        raise ImportError("libdwba_b200.so ABI version mismatch")
    sizes = (ctypes.c_int64 * 18)()
    lib.dwba_struct_sizes(sizes, 18)
    want = (NODESET_DTYPE.itemsize, FOLD_DTYPE.itemsize, FORM_DTYPE.itemsize, TAIL_DTYPE.itemsize,
            FORM_GRAD_DTYPE.itemsize, FOLD_ADJ_DTYPE.itemsize, FOLD_MULTI_DTYPE.itemsize,
            POTENTIAL_DTYPE.itemsize, DOT_DTYPE.itemsize, CUPY_SET_DTYPE.itemsize, CUPY_FORM_DTYPE.itemsize,
            TC_SEGMENT_DTYPE.itemsize, TC_TILE_DTYPE.itemsize, PANEL_COL_DTYPE.itemsize, PANEL_DTYPE.itemsize,
            PANEL_CTA_DTYPE.itemsize, PANEL_ENTRY_DTYPE.itemsize, PANEL_LAYOUT_DTYPE.itemsize)
    if tuple(sizes) != want:
        raise ImportError(f"struct layout mismatch: library {tuple(sizes)} vs binding {want}")
    _lib = lib
    return lib


def status_string(status: int) -> str:
    return load().dwba_status_string(int(status)).decode()


def check(status: int, where: str) -> None:
    if status != DWBA_OK:
        if status == DWBA_ERR_INVALID_ARG:
            raise ValueError(f"{where}: {status_string(status)}")
        raise DWBAError(status, where)


def device_ok() -> bool:
    """True when a usable sm_100 device is visible (the check_cupy_runtime analogue)."""
    lib = load()
    n, ma, mi = ctypes.c_int(0), ctypes.c_int(0), ctypes.c_int(0)
    return lib.dwba_device_probe(ctypes.byref(n), ctypes.byref(ma), ctypes.byref(mi)) == DWBA_OK


def phase_breaks_coulomb(r_start, r_end, k_total, dphi, eta_total):
    lib = load()
    cap = 10010
    out = np.empty(cap, dtype=np.float64)
    n = ctypes.c_int(0)
    check(lib.dwba_phase_breaks_coulomb(float(r_start), float(r_end), float(k_total), float(dphi), float(eta_total),
                                        out.ctypes.data, cap, ctypes.byref(n)), "dwba_phase_breaks_coulomb")
    return out[:n.value].copy()


def tail_on_device(wave, r_m, r_max) -> bool:
    w = np.ascontiguousarray(wave, dtype=np.float64)
    return bool(load().dwba_outer_tail_on_device(w.ctypes.data, float(r_m), float(r_max)))


def tails_on_device(waves: np.ndarray, r_m: np.ndarray, r_max: float) -> np.ndarray:
    """tail_on_device of every row of ``waves`` (n x 10)."""
    w = np.ascontiguousarray(waves, dtype=np.float64)
    m = np.ascontiguousarray(r_m, dtype=np.float64)
    out = np.zeros(len(w), dtype=np.uint8)
    check(load().dwba_outer_tails_on_device(w.ctypes.data, m.ctypes.data, len(w), float(r_max), out.ctypes.data),
          "dwba_outer_tails_on_device")
    return out.astype(bool)


def l0_corrections(chi_i: np.ndarray, chi_f: np.ndarray, n1: np.ndarray, w: np.ndarray, u_i: np.ndarray,
                   u_f: np.ndarray, v_diff: np.ndarray, tol: float):
    """dwba_l0_corrections: (corr_dir, corr_ex) of pairs whose waves (len(w) doubles) lie at the given addresses."""
    f8 = lambda a: np.ascontiguousarray(a, dtype=np.float64)  # noqa: E731
    w, u_i, u_f, v_diff = f8(w), f8(u_i), f8(u_f), f8(v_diff)
    n, N = len(n1), len(w)
    for name, a in (("u_i", u_i), ("u_f", u_f), ("V_core - U_i", v_diff)):
        if a.shape != (N,):
            raise ValueError(f"{name}: shape {a.shape} on a grid of {N} points")
    ci, cf = np.ascontiguousarray(chi_i, dtype=np.uint64), np.ascontiguousarray(chi_f, dtype=np.uint64)
    n1 = np.ascontiguousarray(n1, dtype=np.int64)
    out = np.zeros((2, n))
    check(load().dwba_l0_corrections(ci.ctypes.data, cf.ctypes.data, n1.ctypes.data, n, N, w.ctypes.data,
                                     u_i.ctypes.data, u_f.ctypes.data, v_diff.ctypes.data, float(tol),
                                     out.ctypes.data, out.ctypes.data + 8 * n), "dwba_l0_corrections")
    return out[0], out[1]


def panel_layout(entries: np.ndarray, n_sets: int, n_rows: int, n_trans: int, min_share: float, min_forms: int) -> dict:
    """dwba_panel_layout: its output arrays by name, cut to their counts, and the counts."""
    n = len(entries)
    buf = np.empty((len(PANEL_LAYOUT_ARRAYS), n), dtype=np.int32)
    lay = np.zeros(1, dtype=PANEL_LAYOUT_DTYPE)
    for i, name in enumerate(PANEL_LAYOUT_ARRAYS):
        lay[name] = buf.ctypes.data + 4 * n * i
    check(load().dwba_panel_layout(entries.ctypes.data, n, int(n_sets), int(n_rows), int(n_trans), float(min_share),
                                   int(min_forms), lay.ctypes.data), "dwba_panel_layout")
    out = {c: int(lay[c][0]) for c in ("n_a", "n_b", "n_psi", "n_direct", "n_exchange")}
    a = dict(zip(PANEL_LAYOUT_ARRAYS, buf))
    for names, m in ((("a_u", "a_w", "a_set"), out["n_a"]), (("b_u", "b_w", "b_set"), out["n_b"]),
                     (("psi_t", "psi_set"), out["n_psi"]), (("d_M", "d_F", "d_set"), out["n_direct"]),
                     (("x_M", "x_F", "x_set"), out["n_exchange"])):
        for c in names:
            a[c] = a[c][:m]
    for k in "dx":
        M, F = a[k + "_M"].astype(np.int64), a[k + "_F"].astype(np.int64)
        a[k + "_rows"], a[k + "_entry"] = a[k + "_rows"][:M.sum()], a[k + "_entry"][:(M * F).sum()]
        for c in (("d_psi", "d_wave") if k == "d" else ("x_cols",)):
            a[c] = a[c][:F.sum()]
    return {**out, **a}


def outer_tails(wave, r_m, r_max, L_max, moments, mode, max_filon_segments, max_effective_dphi):
    lib = load()
    w = np.ascontiguousarray(wave, dtype=np.float64)
    m = np.ascontiguousarray(moments, dtype=np.float64)
    out = np.zeros(L_max + 1, dtype=np.float64)
    check(lib.dwba_outer_tails(w.ctypes.data, float(r_m), float(r_max), int(L_max), m.ctypes.data, int(mode),
                               int(max_filon_segments), float(max_effective_dphi), out.ctypes.data),
          "dwba_outer_tails")
    return out
