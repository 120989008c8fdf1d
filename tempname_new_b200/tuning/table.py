"""Tile / raster choices of the dense tcgen05 kernel per problem shape.

The reference keeps one compiled-in C++ record per (meta, shape) under
``src/*/tuning_config/*.cu`` and can load more from ``FLUX_TUNE_CONFIG_FILE``; here the kernel
has three run-time knobs — CTA pairing (``cta_group``), tile width (``tile_n``) and the raster
group (``group_m``) — so the table is a small dict of measured winners plus a heuristic for
unseen shapes. ``python -m tempname_new_b200.tuning.tune_dense`` measures a shape and prints
the entry to add; ``FLUXB_TUNE_FILE`` names a JSON file of extra entries.
"""
from __future__ import annotations

import functools
import json
import os
from typing import Dict, Tuple

Key = Tuple[int, int, int]

# (M rows computed per GPU, N, K) -> knobs. Measured on B200 (148 SMs, 1000 W cap), bf16, with
# `tune_dense --seconds 0.6` (back-to-back launches, so the power cap decides): TFLOP/s of the winner
# and of torch.matmul on the same box in the same process. The key has no element type: 8-bit operands of these shapes get
# the same knobs (measured apart: 16384 x 3584 x 8192 e4m3 407 us, 388 with the heuristic's; int8 344, 353 with them).
DENSE_TABLE: Dict[Key, Dict[str, int]] = {
    # 512 x 256 CTA-pair tiles (two MMAs per k-step share one B tile) win every large shape; the raster
    # group differs: 8 tile rows (4096 rows) unless N is small next to K
    (8192, 49152, 12288): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},   # 1358 | 1400
    (8192, 12288, 49152): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 4},   # 1354 | 1291
    (8192, 24576, 12288): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},   # 1354 | 1388
    (8192, 12288, 24576): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},   # 1333 | 1305
    (8192, 12288, 12288): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},   # 1323 | 1313
    (8192, 6144, 12288): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},    # 1267 | 1316
    (8192, 12288, 6144): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},    # 1291 | 1316
    (16384, 3584, 8192): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 2},    # 1255 | 1272
}

# The same for the fused ops of several ranks (rows of all ranks for all-gather and reduce-scatter): measured before
# the single-GPU rules changed to what is faster there, and kept as they were measured.
MULTI_RANK_TABLE: Dict[Key, Dict[str, int]] = {
    (4096, 4096, 4096): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},
    (4096, 12288, 4096): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},
    (16384, 8192, 3584): {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8},
}

_NUM_SMS = 148


def _wave_eff(tiles: int, slots: int) -> float:
    waves = -(-tiles // slots)
    return tiles / (waves * slots)


def heuristic(m: int, n: int, k: int, elt: int = 2, ranks: int = 1) -> Dict[str, int]:
    """The default of a shape without a measured entry, see ``_heuristic``; ``ranks``: ranks of the fused op."""
    cg, bn, group = _heuristic(m, n, k, elt, ranks)
    return {"cta_group": cg, "tile_n": bn, "group_m": group}


@functools.lru_cache(maxsize=4096)
def _heuristic(m: int, n: int, k: int, elt: int, ranks: int) -> Tuple[int, int, int]:
    """(cta_group, tile_n, group_m); tile_m stays 0: the launcher picks 512-row tiles.

    One rank: CTA pairs on 256 x 256 tiles wherever they need no more waves than single CTAs on 128 x 256 (1000 x
    3000 x 5000 fp16: 41 against 53 us; 1500 x 4000 x 4096 bf16: 52 either way). Raster groups of 2048 rows (with
    wave-synchronous tile starts the grid walks K together, so the group does not have to fit L2 over the whole K
    extent), of 4096 rows for the 256-row tiles of a short K (4096 x 16384 x 4096 bf16 434 -> 416 us, 8192 x 8192 x
    8192 fp8 427 -> 416, never slower by more than the noise).

    Several ranks: pairs unless the problem is too small to fill 74 of them, eight tile rows per group. The tiles of
    a short K have 512 rows there and a group that exceeds a segment's tile rows makes bands span two segments, so
    the single-rank figures do not carry over; these are the choices that the fused ops were measured with."""
    up = lambda a, b: -(-a // b)  # noqa: E731
    t1, t2 = up(m, 128) * up(n, 256), up(m, 256) * up(n, 256)
    fill = m >= 256 and n >= 256 and (m // 256) * up(n, 256) >= _NUM_SMS // 4
    no_more_waves = (ranks == 1 and m >= 256 and n >= 256 and t2 >= _NUM_SMS // 8
                     and up(t2, _NUM_SMS // 2) <= up(t1, _NUM_SMS))
    if fill or no_more_waves:
        cg, bn = 2, 256
    elif n % 256 == 0 or n > 2048:
        cg, bn = 1, 256
    else:
        cg, bn = 1, 128
    group = 16 if cg == 1 or (ranks == 1 and k * elt < 80 * 128) else 8
    return cg, bn, group


def candidates(m: int, n: int, k: int, elt: int = 2, segmented_rows: int = 0):
    """Knob sets worth timing for a dense-kernel problem: 512-row CTA-pair tiles (two MMAs share a B
    tile) where the rows allow them, 256-row CTA pairs, single CTAs; a few raster groups each.
    ``segmented_rows``: rows per rank segment of a fused op (0: plain GEMM over m rows)."""
    rows = segmented_rows or m
    out = []
    if rows >= 512 and n >= 256:
        out += [{"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": g} for g in (2, 4, 8)]
    if rows >= 256 and n >= 256:
        out += [{"cta_group": 2, "tile_n": 256, "tile_m": 256, "group_m": g} for g in (4, 8)]
    out += [{"cta_group": 1, "tile_n": 256 if n >= 256 else 128, "tile_m": 128, "group_m": g} for g in (8, 16)]
    if n % 256:
        out.append({"cta_group": 1, "tile_n": 128, "tile_m": 128, "group_m": 16})
    return out


def _load_extra() -> Dict[Key, Dict[str, int]]:
    path = os.environ.get("FLUXB_TUNE_FILE")
    if not path:
        return {}
    with open(path) as f:
        raw = json.load(f)
    return {tuple(e["key"]): e["best"] for e in raw}


_EXTRA = None
_OVERRIDE: Dict[Key, Dict[str, int]] = {}


class override:
    """``with override((m, n, k), knobs):`` pins the knobs of one shape for the calls inside the
    block - how the tuners try candidates through the public ops."""

    def __init__(self, key: Key, knobs: Dict[str, int]):
        self.key, self.knobs = tuple(key), dict(knobs)

    def __enter__(self):
        self.prev = _OVERRIDE.get(self.key)
        _OVERRIDE[self.key] = self.knobs
        return self

    def __exit__(self, *exc):
        if self.prev is None:
            _OVERRIDE.pop(self.key, None)
        else:
            _OVERRIDE[self.key] = self.prev
        return False


def _entry(key: Key, ranks: int = 1):
    global _EXTRA
    if _EXTRA is None:
        _EXTRA = _load_extra()
    for table in (_OVERRIDE, _EXTRA, DENSE_TABLE):
        if key in table:
            return table[key]
    return MULTI_RANK_TABLE.get(key) if ranks > 1 else None


def lookup(m: int, n: int, k: int, elt: int = 2, ranks: int = 1) -> Dict[str, int]:
    """Knobs of a dense launch of ``m`` rows, for an op whose ``ranks`` ranks take part in one fused launch."""
    e = _entry((m, n, k), ranks)
    return dict(e) if e is not None else heuristic(m, n, k, elt, ranks)


def resolve(m: int, n: int, k: int, elt: int = 2, ranks: int = 1) -> Tuple[int, int, int, int, bool]:
    """``lookup`` for a launch: (cta_group, tile_n, group_m, tile_m, whether a measured or pinned entry answered)."""
    e = _entry((m, n, k), ranks)
    if e is not None:
        return e["cta_group"], e["tile_n"], e["group_m"], e.get("tile_m", 0), True
    return (*_heuristic(m, n, k, elt, ranks), 0, False)
