"""Per-launch figures of an ncu capture, in the machine-readable form bench.py reads.

bench.py reports two numbers it cannot measure inside its own timed region: the
DRAM bytes of one association pass (roofline.traffic) and the warp instructions
that its kernels issue (roofline.issue).  Both come from one `ncu` capture of
the same kernels on a small case of the workload, scaled per pair.  A pass is several
launches (the candidate test and the two launches of the row pass), whose figures are
added up; passes are averaged.  This module turns that capture into
profiles/<kernel>_<workload>.json:

  python -m rkhs_ba_gb300.profiling <capture.ncu-rep> --kernel k_cand,k_rows --launches 3 --pairs 2 \
      --command "<the ncu command that made the capture>" --out profiles/k_rows_global50k.json

It runs `ncu -i <capture> --page raw --csv` (no GPU needed).
"""
from __future__ import annotations

import argparse
import csv
import io
import json
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
METRICS = ("dram__bytes_read.sum", "dram__bytes_write.sum", "smsp__inst_executed.sum", "gpu__time_duration.sum")


# unit strings of the raw page -> bytes or nanoseconds
_SCALE = {"byte": 1.0, "Kbyte": 1e3, "KB": 1e3, "Mbyte": 1e6, "MB": 1e6, "Gbyte": 1e9, "GB": 1e9,
          "nsecond": 1.0, "ns": 1.0, "usecond": 1e3, "us": 1e3, "msecond": 1e6, "ms": 1e6}


def _number(v: str) -> float:
    return float(v.replace(",", ""))


def read_capture(path: str, kernel: str, launches: int = 1) -> dict:
    """METRICS of a pass of `launches` launches of `kernel` (names separated by commas), the
    mean of the captured passes (values in bytes, instructions, nanoseconds)."""
    out = subprocess.run(["ncu", "-i", path, "--page", "raw", "--csv"], check=True, capture_output=True,
                         text=True).stdout
    return read_raw(out, kernel, launches)


def read_raw(text: str, kernel: str, launches: int = 1) -> dict:
    """read_capture of the raw page's text."""
    rows = list(csv.reader(io.StringIO(text)))
    head = rows[0]
    units = rows[1] if len(rows) > 1 else []
    col = {m: head.index(m) for m in METRICS if m in head}
    kcol = head.index("Kernel Name")
    names = kernel.split(",")
    acc = {m: [] for m in col}
    for r in rows[2:]:
        if len(r) <= kcol or not any(n in r[kcol] for n in names):
            continue
        for m, c in col.items():
            u = units[c] if c < len(units) else ""
            acc[m].append(_number(r[c]) * _SCALE.get(u, 1.0))
    for v in acc.values():
        if len(v) % launches:
            raise ValueError("%d launches of %s in the capture, %d to a pass" % (len(v), kernel, launches))
    return {m: sum(v) / (len(v) // launches) for m, v in acc.items() if v}


def summarize(path: str, kernel: str, pairs: int, command: str, launches: int = 1) -> dict:
    m = read_capture(path, kernel, launches)
    dram = m.get("dram__bytes_read.sum", 0.0) + m.get("dram__bytes_write.sum", 0.0)
    return {"kernel": kernel, "launches_per_pass": launches, "pairs_per_launch": pairs, "command": command,
            "dram_bytes_per_pair_launch": round(dram / pairs),
            "warp_instructions_per_pair_launch": round(m.get("smsp__inst_executed.sum", 0.0) / pairs),
            "gpu_time_ns_per_launch": round(m.get("gpu__time_duration.sum", 0.0)),
            "source": os.path.basename(path)}


def load(name: str) -> dict | None:
    """profiles/<name> as a dict, or None when absent."""
    p = os.path.join(ROOT, "profiles", name)
    if not os.path.exists(p):
        return None
    with open(p) as fh:
        return json.load(fh)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("capture")
    ap.add_argument("--kernel", default="k_cand,k_rows", help="kernels of a pass, separated by commas")
    ap.add_argument("--launches", type=int, default=3, help="their launches in a pass")
    ap.add_argument("--pairs", type=int, required=True)
    ap.add_argument("--command", required=True)
    ap.add_argument("--out", required=True)
    a = ap.parse_args()
    d = summarize(a.capture, a.kernel, a.pairs, a.command, a.launches)
    with open(a.out, "w") as fh:
        json.dump(d, fh, indent=1)
        fh.write("\n")
    print(json.dumps(d))


if __name__ == "__main__":
    main()
