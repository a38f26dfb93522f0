#!/usr/bin/env python3
"""Kernel generator front-end for the B200 build.

Keeps the command line of the reference generator
(include/code_gen/scripts/fft_codegen.py:707-736: --if_ft --if_err_injection
--err_smoothing --err_inj --err_threshold --datatype --gpu) and its input, the
per-GPU 11-column parameter CSV (fft_codegen.py:738-752), but emits something
different: the kernels are hand-written templates (csrc/fft_kernels.cuh), so one
pass writes the list of template instantiations a parameter file needs --
csrc/generated/<datatype>/inst_ft<mode>_p<k>.cu with mode 0 (plain), 1 (--if_ft 1)
or 2 (--if_ft 1 --if_err_injection 1), the three passes compile.sh:3-8 runs per
datatype -- plus the parameter table baked into the library
(generated/default_params_<datatype>.inc) and, for FT passes, the default FT
literals (generated/ft_defaults.h; the reference pastes them into the kernel text
at fft_codegen.py:414,495, here they are defaults of run-time arguments).

Extra launches to compile for tuning can be listed in
param/<gpu>/extra_<datatype>.csv (same 11 columns).
"""
from __future__ import annotations

import argparse
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
sys.path.insert(0, os.path.dirname(PKG))
from turbofft_b200.planner import launches_of_row, parse_param_csv  # noqa: E402
from turbofft_b200.codegen import smem_layout  # noqa: E402

# Launches (log2 length, log2 points per thread, log2 lines per tile, role) of rows that a shipped table held until another
# took their place: a caller's own parameter file may hold them, so they stay compiled in every FT mode.
KEPT_LAUNCHES = {"float2": [(5, 3, 5, 0)], "double2": []}

PART_SIZE = 6  # instantiations per translation unit (keeps parallel builds balanced)


def collect_instances(rows):
    seen = []
    for logn in sorted(rows):
        r = rows[logn]
        if r.launches == 0:
            continue
        for l in launches_of_row(r):
            key = (l.logm, l.loge, l.logc, l.role)
            if key not in seen:
                seen.append(key)
    return seen


def narrow_instances(rows, datatype):
    """The multi-launch kernels of the rows again with fewer lines per tile, down to runs of 32 bytes: what
    the planner picks for batches whose tiles would leave SMs without a block (capi.cu, adjust_tiles).
    From 2^22 points on a single signal has tiles enough."""
    least = 2 if datatype == "float2" else 1
    out = []
    for logn in sorted(rows):
        if rows[logn].launches < 2 or logn >= 22:
            continue
        for l in launches_of_row(rows[logn]):
            for logc in range(l.logc - 1, least - 1, -1):
                if (1 << (l.logm - l.loge + logc)) >= 32:
                    out.append((l.logm, l.loge, logc, l.role))
    return out


def write_if_changed(path, text):
    os.makedirs(os.path.dirname(path), exist_ok=True)
    if os.path.exists(path) and open(path).read() == text:
        return False
    with open(path, "w") as f:
        f.write(text)
    return True


def main(argv=None):
    ap = argparse.ArgumentParser(description="turbofft_b200 kernel instantiation generator")
    ap.add_argument("--if_ft", type=int, default=0, help="fault detection (0/1)")
    ap.add_argument("--if_err_injection", type=int, default=0,
                    help="error injection + correction (0/1; 2 = correct from the running checksums, no recompute)")
    ap.add_argument("--err_smoothing", type=int, default=1000, help="additive constant of the detection denominator")
    ap.add_argument("--err_inj", type=int, default=100, help="injected error value")
    ap.add_argument("--err_threshold", type=float, default=1e-3, help="detection threshold")
    ap.add_argument("--datatype", type=str, default="double2", help='"float2" or "double2"')
    ap.add_argument("--gpu", type=str, default="B200", help="GPU spec (directory under param/)")
    ap.add_argument("--out", type=str, default=os.path.join(PKG, "csrc", "generated"))
    args = ap.parse_args(argv)
    if args.datatype not in ("float2", "double2"):
        ap.error("datatype must be float2 or double2")
    if args.if_err_injection:
        args.if_ft = 1
    # --if_err_injection 2 (extension): correction from the running checksums instead of recomputing
    mode = (3 if args.if_err_injection == 2 else 2) if args.if_err_injection else (1 if args.if_ft else 0)

    pdir = os.path.join(PKG, "param", args.gpu)
    csv_text = open(os.path.join(pdir, f"param_{args.datatype}.csv")).read()
    rows = parse_param_csv(csv_text)
    inst = collect_instances(rows)
    inst += [key for key in KEPT_LAUNCHES[args.datatype] if key not in inst]
    extra = os.path.join(pdir, f"extra_{args.datatype}.csv")
    if os.path.exists(extra) and mode == 0:  # tuner candidates are timed with FT off only
        for r in parse_param_csv_multi(open(extra).read()):
            for l in launches_of_row(r):
                key = (l.logm, l.loge, l.logc, l.role)
                if key not in inst:
                    inst.append(key)

    if mode == 0:
        # strided-line kernels of every length 2^1..2^12 for the strided-batch plan
        # (tfft_plan_create_strided), whatever lengths the launch rows above happen to use, and narrower
        # tiles of the rows' own kernels
        for key in STRIDED_LINES[args.datatype] + narrow_instances(rows, args.datatype):
            if key not in inst:
                inst.append(key)
    if mode == 3:
        # checksum-based correction exists for single and last launches of 32 points and more
        inst = [(logm, loge, logc, role) for (logm, loge, logc, role) in inst if role != 1 and logm >= 5]
    ctype = "float" if args.datatype == "float2" else "double"
    dt = 0 if args.datatype == "float2" else 1
    odir = os.path.join(args.out, args.datatype)
    os.makedirs(odir, exist_ok=True)
    prefix = f"inst_ft{mode}_p"
    written = []
    for k in range(0, len(inst), PART_SIZE):
        lines = [
            "// Generated by codegen/fft_codegen.py -- do not edit.",
            f"// datatype={args.datatype} gpu={args.gpu} if_ft={args.if_ft} if_err_injection={args.if_err_injection}",
            '#include "../../instances.cuh"',
        ]
        for (logm, loge, logc, role) in inst[k : k + PART_SIZE]:
            lines.append(f"TFFT_INST({ctype}, {dt}, {logm}, {loge}, {logc}, {role}, {mode})")
        name = f"{prefix}{k // PART_SIZE}.cu"
        write_if_changed(os.path.join(odir, name), "\n".join(lines) + "\n")
        written.append(name)
    for old in os.listdir(odir):  # parts of an earlier, longer list
        if old.startswith(prefix) and old.endswith(".cu") and old not in written:
            os.remove(os.path.join(odir, old))

    # bank-conflict-free shared-memory layouts for this datatype's instances
    cache = smem_layout.load_cache()
    before = {k: list(v) for k, v in cache.items()}
    for (logm, loge, logc, role) in inst:
        smem_layout.best_layout(role, logm, loge, logc, dt == 1, cache)
    if cache != before:
        smem_layout.save_cache(cache)
    lay = ["// Generated by codegen/fft_codegen.py -- shared-memory layouts found by codegen/smem_layout.py.",
           "// SmemLayout<T, LOGM, LOGE, LOGC, ROLE>: pad(a) = a + (a >> PADSHIFT), row pitch = pad(M-1)+1+EXTRA;",
           "// REMLAST = 1 puts the remainder radix into the last register stage instead of the first."]
    for key in sorted(cache):
        f64, role, logm, loge, logc = (int(t) for t in key.split("_"))
        ps, ex = cache[key][:2]
        rl = cache[key][2] if len(cache[key]) > 2 else 0
        lay.append(f"template <> struct SmemLayout<{'double' if f64 else 'float'}, {logm}, {loge}, {logc}, {role}> "
                   f"{{ static constexpr int PADSHIFT = {ps}, EXTRA = {ex}, REMLAST = {rl}; }};")
    write_if_changed(os.path.join(args.out, "smem_layouts.h"), "\n".join(lay) + "\n")

    lit = "".join('"' + ln.strip() + '\\n"\n' for ln in csv_text.splitlines() if ln.strip())
    write_if_changed(os.path.join(args.out, f"default_params_{args.datatype}.inc"), lit)
    # sizes that run as one cluster kernel: "logN, log2 cluster size" (a missing file = none)
    sp = os.path.join(pdir, f"single_pass_{args.datatype}.csv")
    sp_text = open(sp).read() if os.path.exists(sp) else ""
    sp_lit = "".join('"' + ln.strip() + '\\n"\n' for ln in sp_text.splitlines() if ln.strip() and not ln.strip().startswith("#")) or '""\n'
    write_if_changed(os.path.join(args.out, f"default_single_pass_{args.datatype}.inc"), sp_lit)
    # thread_bs a plan created with thread_bs = 0 uses: "logN, FT off, FT on"
    tb = os.path.join(pdir, f"thread_bs_{args.datatype}.csv")
    tb_text = open(tb).read() if os.path.exists(tb) else ""
    tb_lit = "".join('"' + ln.strip() + '\\n"\n' for ln in tb_text.splitlines() if ln.strip() and not ln.strip().startswith("#")) or '""\n'
    write_if_changed(os.path.join(args.out, f"default_thread_bs_{args.datatype}.inc"), tb_lit)
    defaults = os.path.join(args.out, "ft_defaults.h")
    if args.if_ft or not os.path.exists(defaults):
        write_if_changed(
            defaults,
            "// Generated by codegen/fft_codegen.py -- default FT literals (run-time overridable).\n"
            "#pragma once\n"
            f"#define TFFT_DEFAULT_ERR_INJ {float(args.err_inj)!r}\n"
            f"#define TFFT_DEFAULT_ERR_SMOOTHING {float(args.err_smoothing)!r}\n"
            f"#define TFFT_DEFAULT_ERR_THRESHOLD {float(args.err_threshold)!r}\n",
        )
    print(f"[fft_codegen] {args.datatype} mode {mode}: {len(inst)} kernels in {len(written)} files -> {odir}")
    return 0


# (log2 length, log2 points per thread, log2 adjacent columns per tile, ROLE_FIRST): a wide tile
# per length, plus tiles of 4 columns and of 1 column for arrays whose inner extent is smaller
def _narrow(rows):
    out = list(rows)
    for (m, e, c, r) in rows:
        for cc in (2, 0):
            if cc < c and (m, e, cc, r) not in out:
                out.append((m, e, cc, r))
    return out


STRIDED_LINES = {
    "float2": [(1, 1, 5, 1), (2, 2, 5, 1), (3, 3, 5, 1), (4, 4, 5, 1), (5, 4, 5, 1), (6, 4, 4, 1), (7, 4, 5, 1), (8, 4, 4, 1),
               (9, 5, 4, 1), (10, 5, 3, 1), (11, 4, 2, 1), (12, 4, 1, 1)],
    "double2": [(1, 1, 5, 1), (2, 2, 5, 1), (3, 3, 5, 1), (4, 4, 4, 1), (5, 4, 4, 1), (6, 4, 4, 1), (7, 4, 4, 1), (8, 4, 4, 1),
                (9, 4, 3, 1), (10, 4, 2, 1), (11, 4, 1, 1), (12, 4, 0, 1)],
}
STRIDED_LINES = {k: _narrow(v) for k, v in STRIDED_LINES.items()}


def parse_param_csv_multi(text):
    """Rows of an extra_<datatype>.csv: several rows may share a logN."""
    from turbofft_b200.planner import ParamRow

    out = []
    for line in text.splitlines():
        s = line.strip()
        if not s or s.startswith("#"):
            continue
        tok = [int(t) for t in s.split(",")]
        out.append(ParamRow(tok[0], tok[1], tuple(tok[2:5]), tuple(tok[5:8]), tuple(tok[8:11])))
    return out


if __name__ == "__main__":
    sys.exit(main())
