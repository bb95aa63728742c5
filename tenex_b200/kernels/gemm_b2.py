"""GEMM-B2 kernel class: binary (b_max = 2) TE as a tensor-core contraction.

Reference: tenex/kernels/gemm_b2.py (GEMMB2Kernel :565-596, compute_te_gemm_b2
:307-425). Same name, supports() predicate and compute_matrix() contract
([i, j] = TE(j -> i), diagonal 0); the counts come from tcgen05 MMAs over the
0/1 operands, packed as 4-bit E2M1 values (kind::mxf4, float32 sums) or as int8
(kind::i8, int32 sums), both exact, and the 8-cell TE from the TMEM epilogue of
the same kernel (gemm_b2.cu).
"""
from __future__ import annotations

import numpy as np
import torch

from tenex_b200 import native
from tenex_b200.kernels import TEKernel
from tenex_b200.kernels import device as D


OPERANDS = {"default": 0, "int8": 1, "fp4": 2}


TILE_N = (128, 112, 96, 80, 64)


def te_binary_matrix(db: D.DeviceBins, tau: int = 1, out: torch.Tensor | None = None,
                     check: bool = True, operands: str = "default",
                     tile_n: int = 0) -> torch.Tensor:
    """(n, n) float32 device matrix with [src, tgt] = TE(src -> tgt), diagonal 0.
    operands: "int8" (kind::i8 MMAs), "fp4" (the 0/1 values as packed E2M1,
    kind::mxf4) or "default" (fp4); the counts and TE are the same.
    tile_n: targets per GEMM tile, 0 = chosen from n and the SM count
    (tile_width), else one of TILE_N (the same matrix bit for bit)."""
    if tile_n and tile_n not in TILE_N:
        raise ValueError(f"tile_n={tile_n}: expected 0 or one of {TILE_N}")
    dev = db.data.device
    n = db.n
    lag = tau * db.K
    if out is None:
        out = torch.zeros((n, n), dtype=torch.float32, device=dev)
    nb = int(native.lib().tenex_b2_workspace_bytes(n, db.row_len, lag))
    ws = torch.empty(nb, dtype=torch.uint8, device=dev)
    s = native.stream_ptr()
    native.call("tenex_te_binary_matrix_ex", db.ptr(), db.ld, n, db.row_len, lag,
                out.data_ptr(), n, ws.data_ptr(), nb, OPERANDS[operands], int(tile_n), s)
    if check:
        native.call("tenex_b2_status", ws.data_ptr(), n, db.row_len, lag, s)
    return out


def tile_width(n: int) -> int:
    """Targets per GEMM tile that te_binary_matrix picks for n genes on the
    current device."""
    import ctypes
    tn = ctypes.c_int()
    native.call("tenex_b2_tile_n", int(n), ctypes.byref(tn))
    return tn.value


class GEMMB2Kernel(TEKernel):
    """Exact binary TE for all pairs from three tensor-core contractions (4-bit or
    INT8 operands)."""

    @property
    def name(self) -> str:
        return "GEMM-B2"

    @property
    def is_matrix_kernel(self) -> bool:
        return True

    def supports(self, b_max, on_cuda, smem_optin, smem_bytes, n_per_var,
                 source_filter) -> bool:
        return bool(on_cuda) and b_max == 2 and not source_filter

    def compute_matrix_device(self, db: D.DeviceBins, tau: int) -> torch.Tensor:
        """[src, tgt] = TE(src -> tgt) on the device."""
        return te_binary_matrix(db, tau)

    def compute_matrix(self, data, n_vars: int, tau: int, device, **kwargs) -> np.ndarray:
        dev = torch.device(device) if not isinstance(device, torch.device) else device
        db = D.pack_bins(data, dev, 2)
        if db.K != 1:
            raise ValueError(f"GEMM-B2 kernel only supports K=1, got K={db.K}")
        m = te_binary_matrix(db, tau)
        return D.to_host(m.t())  # reference orientation: [i, j] = TE(j -> i)

    def compute_single_gpu(self, bin_arrs, pairs, b_max, n_per_var, tau, batch_size, device,
                           **kwargs) -> np.ndarray:
        te = self.compute_matrix(bin_arrs, None, tau, device)
        p = pairs.cpu().numpy() if isinstance(pairs, torch.Tensor) else np.asarray(pairs)
        return te[p[:, 0], p[:, 1]]

    def compute_matrix_multi_gpu(self, data, n_vars: int, tau: int, device_ids: list,
                                 **kwargs) -> np.ndarray:
        """Multi-device entry of the reference (tenex/kernels/gemm_b2.py:591-593). The
        binary matrix of 2,000 genes x 5,000 cells takes ~0.1 ms on one B200, so it runs
        on the first listed device."""
        ids = [int(d) for d in device_ids]
        if not ids:
            raise ValueError("device_ids must name at least one device")
        return self.compute_matrix(data, n_vars, tau, torch.device("cuda", ids[0]), **kwargs)

    def log_description(self, **kwargs) -> str:
        return "GEMM-B2 (tcgen05 contractions + fused TE epilogue, exact)"
