"""Plumbing shared by the capture modules."""

from __future__ import annotations

import json
import os
import pathlib
import shutil

ENV_VAR = "MOSAICIST_KNOBS"          # src/mosaicist/converge/knobs.py:21
DUMP_VAR = "MOSAIC_GPU_DUMP_TO"      # src/mosaicist/capture.py:41-47


def from_env(defaults: dict | None = None) -> dict:
    """The knob setting for this capture: JSON in $MOSAICIST_KNOBS merged over `defaults`
    (same contract as mosaicist.converge.knobs.from_env, knobs.py:25-36)."""
    out = dict(defaults or {})
    raw = os.environ.get(ENV_VAR)
    if raw:
        out.update(json.loads(raw))
    return out


def drop_artifacts(*sources: str) -> None:
    """Copies the CUDA sources of the kernels that can run (file names under csrc/) and the ptxas
    log into the capture's dump directory, where collect_artifacts looks for a ptxas-named log
    (capture.py:81-116).  Compiler output of the kernels (PTX, SASS) is neither kept nor read."""
    dump = os.environ.get(DUMP_VAR)
    if not dump:
        return
    from .. import _lib

    dst = pathlib.Path(dump)
    dst.mkdir(parents=True, exist_ok=True)
    for name in sources:
        shutil.copy(_lib.PKG / "csrc" / name, dst / name)
    log = _lib.LIB_PATH.with_suffix(".ptxas.log")
    if log.exists():
        shutil.copy(log, dst / "ptxas_mosaicist_sm100a.log")
