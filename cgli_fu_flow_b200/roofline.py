"""Roofline bookkeeping of the dominant kernel (the wavefront sweep passes).

Algorithmic bytes of one sweep pass per cell: what the four passes of an inner
iteration cannot do without, given the record + MR slot of 16 words that the
residual leaves per cell, over four.  A forward pass reads the slot and writes
its result (16 + 5 words); a backward pass reads the slot and that result; the
last one writes its own (16 + 5 + 5), the first sweep's stores only the halo
planes (16 + 5).  Together 89 words, a mean of 178 B (FP64) or 89 B (CGLI_MIXED)
per pass; on a general grid every pass also reads nine metric words.  The bound
is HBM bandwidth (no dense contraction); the peak is the measured copy bandwidth
of this GPU type (MEASURED_PEAKS.json, the burst figure, since the pass is
timed alone), else 6650 GB/s, an earlier measurement on the same hardware.
"""
from __future__ import annotations

import json
import os

HERE = os.path.dirname(os.path.abspath(__file__))
PEAKS = os.path.join(os.path.dirname(HERE), "MEASURED_PEAKS.json")

SWEEP_WORDS_PER_CELL = (21 + 21 + 21 + 26) / 4
GENERAL_METRIC_WORDS = 9
WORD_BYTES = {"fp64": 8, "mixed": 4}

# DRAM bytes (read + write) per cell of one sweep pass from an ncu capture of
# k_sweep (dram__bytes_read.sum + dram__bytes_write.sum, mean of the four
# passes of an inner iteration: FP64 forward 165 / 165, backward 181 (only the
# halo planes are stored) / 213; FP32 80 / 80, 91 / 103) on the 160x128x128
# channel; traffic grows with the cell count, so it is scaled to the benchmark
# grid.  Channel metrics only.
MEASURED_TRAFFIC_PER_CELL = {"fp64": (165 + 181 + 165 + 213) / 4, "mixed": (80 + 91 + 80 + 103) / 4}


def sweep_bytes_per_cell(precision: str, general: bool = False) -> float:
    return (SWEEP_WORDS_PER_CELL + (GENERAL_METRIC_WORDS if general else 0)) * WORD_BYTES[precision]


def hbm_peak() -> tuple[float, str]:
    try:
        with open(PEAKS) as fh:
            return float(json.load(fh)["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def sweep_roofline(ch, pass_ms: float, precision: str) -> dict:
    """pass_ms: mean device time of one wavefront pass."""
    cells = ch.cells
    bpc = sweep_bytes_per_cell(precision, ch.wavy)
    dur_ms = pass_ms
    achieved = bpc * cells / (dur_ms / 1e3) / 1e9
    peak, kind = hbm_peak()
    tpc = None if ch.wavy else MEASURED_TRAFFIC_PER_CELL.get(precision)
    return {"kernel": "k_sweep (LU-SGS wavefront pass, forward/backward mean)", "bound": "hbm",
            "achieved": round(achieved, 1), "peak": peak, "peak_kind": kind, "unit": "GB/s",
            "frac": round(achieved / peak, 4), "traffic": None if tpc is None else int(tpc * cells),
            "algorithmic_bytes_per_launch": int(bpc * cells), "launch_ms": round(dur_ms, 4)}


# Algorithmic bytes of the residual side of one inner iteration per cell
# (halo and boundaries, the three flux sweeps, the viscous terms and the
# residual assembly together), the per-unit figure of the hot-path scope:
# Q at three time levels (15), J and nine cell metrics (10), three face sets
# of J_f and nine metrics (30), written MR (5): 60 doubles = 480 B.
RESIDUAL_BYTES_PER_CELL = 60 * 8
RESIDUAL_STAGES = ("halo_bc", "flux_x", "flux_y", "flux_z", "viscous", "residual")


# FP64 instructions per cell (thread level) of the residual side's kernels,
# from ncu (sm__inst_executed_pipe_fp64.sum x 32 / cells) on the
# 160x128x128 channel: fluxes 272 / 284 / 293 per face (x / y / z), the viscous
# terms 335, residual assembly 260.  With the FP64 pipe's measured rate on this
# GPU (a standalone FMA probe: 34 TFLOP/s = 17 T FP64 instructions/s) this is a
# lower bound on the side's time.
RESIDUAL_FP64_OPS_PER_CELL = 272 + 284 + 293 + 335 + 260
FP64_INST_PER_S = 17.0e12


def residual_roofline(ch, stage_ms: dict) -> dict:
    """stage_ms: device milliseconds per stage of one inner iteration."""
    dur_ms = sum(stage_ms[k] for k in RESIDUAL_STAGES)
    achieved = RESIDUAL_BYTES_PER_CELL * ch.cells / (dur_ms / 1e3) / 1e9
    fp64_ms = RESIDUAL_FP64_OPS_PER_CELL * ch.cells / FP64_INST_PER_S * 1e3
    peak, kind = hbm_peak()
    return {"kernels": "halo/boundaries, k_flux_x/y/z, k_viscous, k_residual_fast",
            "bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "peak_kind": kind, "unit": "GB/s",
            "frac": round(achieved / peak, 4), "algorithmic_bytes_per_iteration": RESIDUAL_BYTES_PER_CELL * ch.cells,
            "ms_per_iteration": round(dur_ms, 4),
            "fp64_floor_ms": round(fp64_ms, 4), "fp64_frac": round(fp64_ms / dur_ms, 4)}

