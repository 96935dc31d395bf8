#!/usr/bin/env python3
"""Generates `tests/golden/blackwell_golden.npz`: outputs of the REFERENCE's own Blackwell kernels
(per-tensor FP8, MXFP8, NVFP4 quantizers / packers / fused producers and CUTLASS GEMMs) on seeded
inputs, run on a B200, plus a report that compares them with this library's kernels and times
both GEMMs on the same GPU.

Needs a B200 and the reference's extensions compiled by `oracle/build_ref_kernels.py`
(`oracle/_ref/libref_{fp8,mxfp8,fp4}.so`).  Single-GPU only.

    python tests/golden/make_blackwell_golden.py <output-dir> [--ext | --silu]

writes `<output-dir>/blackwell_golden.npz` (copy it to `tests/golden/`) and
`<output-dir>/blackwell_reference_report.json`; with `--ext` the second fixture file
`blackwell_golden_ext.npz` (W4A8-MX, the FP8 producer GEMM, SwiGLU chains) and its report; with
`--silu` the third, `blackwell_golden_silu.npz` (the table-SiLU SwiGLU producer for MXFP8).

Inputs are regenerated by the tests from the same seeds (`case_inputs`), so only outputs are
stored: small cases in full; full-size cases as SHA-256 digests of the code / scale-factor
arrays, the positions where the reference's fast-math build differs from this library's
IEEE-arithmetic kernels (with the reference's value there), and a fixed sample of every GEMM output.
"""

import hashlib
import json
import sys
import time
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[2]
for entry in (str(ROOT), str(ROOT / "robotics-the-speedup-paradox_b200")):
    if entry not in sys.path:
        sys.path.insert(0, entry)

# (name, m, n, k): activation rows, weight rows, reduction length
CASES = (
    ("small", 100, 256, 512),
    ("cfg3_gate_up", 816, 16384, 2048),
    ("cfg4_down", 816, 2048, 16384),
    ("cfg4_q", 816, 2048, 2048),
    ("cfg4_kv", 816, 256, 2048),
)
FULL = ("small",)          # cases whose arrays are stored in full
MAX_LISTED = 65536          # differing positions listed per array at most
SAMPLE_ROWS = (0, 1, 2, 3, 100, 407, 808, 813, 814, 815)
SAMPLE_COL_STEP = 61


def case_inputs(name, m, n, k):
    """Seeded bf16 inputs of a case (CPU generator: identical on every machine)."""
    seed = 1000 + sum(ord(c) for c in name)
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k, generator=gen).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=gen) * 0.02).to(torch.bfloat16)
    bias = (torch.randn(n, generator=gen) * 0.01).to(torch.bfloat16)
    return x, w, bias


def producer_inputs(rows=100, k=512, inter=768):
    gen = torch.Generator().manual_seed(77)
    x = torch.randn(rows, k, generator=gen).to(torch.bfloat16)
    res = torch.randn(rows, k, generator=gen).to(torch.bfloat16)
    weight = (1.0 + 0.1 * torch.randn(k, generator=gen)).to(torch.bfloat16)
    gate_up = (torch.randn(rows, 2 * inter, generator=gen) * 2.0).to(torch.bfloat16)
    return x, res, weight, gate_up, inter


def sha(array):
    return hashlib.sha256(np.ascontiguousarray(array).tobytes()).hexdigest()


def sample_rows(m):
    return np.array([r for r in SAMPLE_ROWS if r < m], dtype=np.int64)


def out_sample(out):
    """Fixed sample of a [m, n] bf16 output as uint16 bit patterns."""
    rows = sample_rows(out.shape[0])
    return out[rows][:, ::SAMPLE_COL_STEP].contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def diff_listing(ref, ours):
    """Positions (flat) where two uint8 arrays differ, with the reference's bytes there."""
    ref, ours = np.asarray(ref).reshape(-1), np.asarray(ours).reshape(-1)
    pos = np.nonzero(ref != ours)[0]
    return int(pos.size), pos[:MAX_LISTED].astype(np.int64), ref[pos[:MAX_LISTED]].astype(np.uint8)


def store_array(store, key, ref, ours, full):
    """Digest (+ full copy for small cases) of a reference array, and its difference to ours."""
    ref_np = ref.contiguous().view(torch.uint8).cpu().numpy()
    ours_np = ours.contiguous().view(torch.uint8).cpu().numpy()
    store[key + "_sha"] = np.array(sha(ref_np))
    if full:
        store[key] = ref_np
    count, pos, val = diff_listing(ref_np, ours_np)
    store[key + "_diff_count"] = np.array(count, dtype=np.int64)
    store[key + "_diff_pos"] = pos
    store[key + "_diff_val"] = val
    return count, ref_np.size


def time_us(fn, reps=20, inner=10):
    """Microseconds per call: CUDA events around `reps` replays of a graph of `inner` calls; falls
    back to eager back-to-back launches when the op cannot be captured."""
    for _ in range(3):
        fn()
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    graph = None
    try:
        graph = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        side.wait_stream(stream)
        with torch.cuda.graph(graph, stream=side):
            for _ in range(inner):
                fn()
        stream.wait_stream(side)
        graph.replay()
        torch.cuda.synchronize()
    except Exception:  # noqa: BLE001 - any capture failure selects the eager loop
        graph = None
        torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(reps):
        if graph is not None:
            graph.replay()
        else:
            for _ in range(inner):
                fn()
    b.record()
    torch.cuda.synchronize()
    return a.elapsed_time(b) / (reps * inner) * 1e3, ("graph" if graph is not None else "eager")


def compare_out(ref, ours):
    r, o = ref.float(), ours.float()
    rel = float((o - r).norm() / r.norm())
    unequal = int((ref.view(torch.int16) != ours.view(torch.int16)).sum().item())
    return {"rel_frobenius": rel, "max_abs": float((o - r).abs().max().item()), "bf16_unequal": unequal,
            "elements": ref.numel()}


def main(out_dir):
    from oracle import blockscale as OB
    from oracle import ref_kernels as RK
    from rk_b200 import fp4_linear as P4
    from rk_b200 import fp8_linear as P8

    dev = torch.device("cuda:0")
    torch.cuda.set_device(0)
    store, report = {}, {"device": torch.cuda.get_device_name(0), "cases": {}, "producers": {}, "timing_us": {}}
    ops = {}
    for backend in ("fp8", "mxfp8", "fp4"):
        ns, why = RK.load(backend)
        ops[backend] = ns
        report[backend + "_extension"] = "loaded" if ns is not None else f"unavailable: {why}"
        print(backend, report[backend + "_extension"], flush=True)

    for name, m, n, k in CASES:
        full = name in FULL
        x, w, bias = (t.to(dev) for t in case_inputs(name, m, n, k))
        entry = report["cases"].setdefault(name, {"m": m, "n": n, "k": k})
        timing = report["timing_us"].setdefault(name, {})

        # ---------------------------------------------------------------- per-tensor FP8
        if ops["fp8"] is not None:
            o = ops["fp8"]
            ra, rsa = o.quantize_bf16(x)
            rb, rsb = o.quantize_bf16(w)
            oa, osa = P8.quantize_bf16(x)
            ob, osb = P8.quantize_bf16(w)
            store[f"{name}_fp8_a_scale"] = rsa.reshape(1).cpu().numpy()
            store[f"{name}_fp8_w_scale"] = rsb.reshape(1).cpu().numpy()
            ca = store_array(store, f"{name}_fp8_a_codes", ra, oa, full)
            cb = store_array(store, f"{name}_fp8_w_codes", rb, ob, full)
            entry["fp8"] = {"a_codes_differ": ca, "w_codes_differ": cb,
                            "a_scale_equal": bool(rsa.item() == osa.item()), "w_scale_equal": bool(rsb.item() == osb.item())}
            # GEMMs on the REFERENCE's codes and scales, both libraries
            rsa1, rsb1 = rsa.reshape(1), rsb.reshape(1)
            mine = P8.linear_forward_packed(ra, rsa1, rb, rsb1, bias)
            store[f"{name}_fp8_out_ours_sample"] = out_sample(mine)
            for tactic in (1, 6, 2):  # 128x128x64 one CTA; 128x256x128 one CTA; 256x128x64 CTA pair
                try:
                    ref = o.linear_forward_packed_tactic(ra, rsa1, rb, rsb1, bias, tactic)
                    torch.cuda.synchronize()
                except RuntimeError as error:
                    entry["fp8"][f"gemm_t{tactic}"] = f"failed: {str(error)[:200]}"
                    continue
                entry["fp8"][f"gemm_t{tactic}"] = compare_out(ref, mine)
                store[f"{name}_fp8_out_t{tactic}_sample"] = out_sample(ref)
                if full:
                    store[f"{name}_fp8_out_t{tactic}"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
                timing[f"fp8_ref_t{tactic}"] = time_us(lambda: o.linear_forward_packed_tactic(ra, rsa1, rb, rsb1, bias, tactic))
            timing["fp8_ours"] = time_us(lambda: P8.linear_forward_packed(ra, rsa1, rb, rsb1, bias))
            print(name, "fp8", entry["fp8"], timing, flush=True)

        # ---------------------------------------------------------------- MXFP8
        if ops["mxfp8"] is not None:
            o = ops["mxfp8"]
            ra, rfa = o.pack(x)
            rb, rfb = o.pack(w)
            oa, ofa = P8.mxfp8_pack(x)
            ob, ofb = P8.mxfp8_pack(w)
            entry["mxfp8"] = {
                "a_codes_differ": store_array(store, f"{name}_mxfp8_a_codes", ra, oa, full),
                "a_sf_differ": store_array(store, f"{name}_mxfp8_a_sf", rfa, ofa, full),
                "w_codes_differ": store_array(store, f"{name}_mxfp8_w_codes", rb, ob, full),
                "w_sf_differ": store_array(store, f"{name}_mxfp8_w_sf", rfb, ofb, full),
            }
            mine = P8.mxfp8_linear(ra, rfa, rb, rfb, bias)
            store[f"{name}_mxfp8_out_ours_sample"] = out_sample(mine)
            tactics = [1, 6] + ([102, 2, 4] if n % 256 == 0 else [])
            for tactic in tactics:  # 128x128x128 c1; 128x256x128 c1; 256x256x128 CTA pairs (102 = the caller's)
                try:
                    ref = o.linear(ra, rfa, rb, rfb, bias, tactic)
                    torch.cuda.synchronize()
                except RuntimeError as error:
                    entry["mxfp8"][f"gemm_t{tactic}"] = f"failed: {str(error)[:200]}"
                    continue
                entry["mxfp8"][f"gemm_t{tactic}"] = compare_out(ref, mine)
                store[f"{name}_mxfp8_out_t{tactic}_sample"] = out_sample(ref)
                if full:
                    store[f"{name}_mxfp8_out_t{tactic}"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
                timing[f"mxfp8_ref_t{tactic}"] = time_us(lambda: o.linear(ra, rfa, rb, rfb, bias, tactic))
            timing["mxfp8_ours"] = time_us(lambda: P8.mxfp8_linear(ra, rfa, rb, rfb, bias))
            print(name, "mxfp8", entry["mxfp8"], timing, flush=True)

        # ---------------------------------------------------------------- NVFP4 (no per-tensor scale: the reference's format)
        if ops["fp4"] is not None:
            o = ops["fp4"]
            ra, rfa = o.pack_activation_gemm_bf16(x)
            rb, rfb, meta = o.pack_linear_weight_gemm_bf16(w, "linear", name)
            oa, ofa = P4.pack_nvfp4(x)
            ob, ofb = P4.pack_nvfp4(w)
            # the reference leaves the padding bytes of the activation scale buffer uninitialised
            # (rows beyond m inside the last 128-row block): zero them, as this library writes them
            valid = torch.zeros(ofa.numel(), dtype=torch.bool, device=dev)
            valid[torch.from_numpy(OB.sf_offsets(m, k // 16).reshape(-1)).to(dev)] = True
            rfa = torch.where(valid, rfa.reshape(-1), torch.zeros_like(ofa)).reshape(rfa.shape)
            entry["nvfp4"] = {
                "a_codes_differ": store_array(store, f"{name}_nvfp4_a_codes", ra, oa, full),
                "a_sf_differ": store_array(store, f"{name}_nvfp4_a_sf", rfa.reshape(-1), ofa, full),
                "w_codes_differ": store_array(store, f"{name}_nvfp4_w_codes", rb, ob, full),
                "w_sf_differ": store_array(store, f"{name}_nvfp4_w_sf", rfb.reshape(-1), ofb, full),
            }
            rfa1, rfb1 = rfa.reshape(-1).contiguous(), rfb.reshape(-1).contiguous()
            mine = P4.linear_forward_packed_gemm_bf16(ra, rfa1, None, rb, rfb1, None, bias, k)
            mine_nobias = P4.linear_forward_packed_gemm_bf16(ra, rfa1, None, rb, rfb1, None, None, k)
            store[f"{name}_nvfp4_out_ours_sample"] = out_sample(mine)
            # 0 = the reference's own choice (bias fused); 1 = 256x256x256, 3 = 256x192x256 CTA pairs: these two
            # specialisations have no bias in their epilogue, so they are compared without one
            for tactic in (0, 1, 3):
                tb = bias if tactic == 0 else None
                try:
                    ref = o.linear_forward_packed_gemm_bf16_tactic(ra, rfa, rb, rfb, meta, tb, "linear", name, tactic)
                    torch.cuda.synchronize()
                except RuntimeError as error:
                    entry["nvfp4"][f"gemm_t{tactic}"] = f"failed: {str(error)[:200]}"
                    continue
                entry["nvfp4"][f"gemm_t{tactic}"] = compare_out(ref, mine if tactic == 0 else mine_nobias)
                store[f"{name}_nvfp4_out_t{tactic}_sample"] = out_sample(ref)
                if full:
                    store[f"{name}_nvfp4_out_t{tactic}"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
                timing[f"nvfp4_ref_t{tactic}"] = time_us(
                    lambda: o.linear_forward_packed_gemm_bf16_tactic(ra, rfa, rb, rfb, meta, tb, "linear", name, tactic))
            timing["nvfp4_ours"] = time_us(lambda: P4.linear_forward_packed_gemm_bf16(ra, rfa1, None, rb, rfb1, None, bias, k))
            print(name, "nvfp4", entry["nvfp4"], timing, flush=True)
        del x, w
        torch.cuda.empty_cache()

    # -------------------------------------------------------------------- fused producers (small)
    x, res, weight, gate_up, inter = (t.to(dev) if torch.is_tensor(t) else t for t in producer_inputs())
    eps = 1e-6
    if ops["fp8"] is not None:
        o = ops["fp8"]
        rs, rn, rq, rscale = o.add_rms_norm_quantize_bf16(x, res, weight, eps)
        os_, on, oq, oscale = P8.add_rms_norm_quantize_bf16(x, res, weight, eps)
        report["producers"]["fp8_rmsnorm"] = {
            "sum_differ": store_array(store, "prod_fp8_rms_sum", rs, os_, True),
            "norm_differ": store_array(store, "prod_fp8_rms_norm", rn, on, True),
            "codes_differ": store_array(store, "prod_fp8_rms_codes", rq, oq, True),
            "scale_equal": bool(rscale.item() == oscale.item())}
        store["prod_fp8_rms_scale"] = rscale.reshape(1).cpu().numpy()
        rq, rscale = o.quantize_swiglu_bf16(gate_up, inter)
        oq, oscale = P8.quantize_swiglu_bf16(gate_up, inter)
        report["producers"]["fp8_swiglu"] = {"codes_differ": store_array(store, "prod_fp8_swiglu_codes", rq, oq, True),
                                             "scale_equal": bool(rscale.item() == oscale.item())}
        store["prod_fp8_swiglu_scale"] = rscale.reshape(1).cpu().numpy()
    if ops["fp4"] is not None:
        o = ops["fp4"]
        outs = o.add_rms_norm_fp4_quant_bf16(x, res, weight, eps, True)
        os_, on, oq, osf = P4.add_rms_norm_fp4_quant_bf16(x, res, weight, eps, True)
        report["producers"]["nvfp4_rmsnorm_outputs"] = [list(t.shape) for t in outs]
        names = ("sum", "norm", "codes", "sf") if len(outs) == 4 else ("sum", "codes", "sf")
        # the reference leaves the padding bytes of this scale buffer uninitialised: keep the valid ones only
        valid = torch.zeros(osf.numel(), dtype=torch.bool, device=dev)
        valid[torch.from_numpy(OB.sf_offsets(x.shape[0], x.shape[1] // 16).reshape(-1)).to(dev)] = True
        outs = list(outs)
        outs[-1] = torch.where(valid, outs[-1].reshape(-1), torch.zeros_like(osf))
        mine = {"sum": os_, "norm": on, "codes": oq, "sf": torch.where(valid, osf, torch.zeros_like(osf))}
        report["producers"]["nvfp4_rmsnorm"] = {
            key + "_differ": store_array(store, "prod_nvfp4_rms_" + key, t.reshape(-1), mine[key].reshape(-1), True)
            for key, t in zip(names, outs)}
        for interleaved in (False, True):
            act = o.silu_mul_bf16(gate_up, inter, interleaved)
            store[f"prod_nvfp4_silu_mul_{int(interleaved)}"] = act.view(torch.int16).cpu().numpy().view(np.uint16)
    print(json.dumps(report["producers"]), flush=True)

    out_dir = Path(out_dir)
    out_dir.mkdir(parents=True, exist_ok=True)
    store["generated"] = np.array(time.strftime("%Y-%m-%d") + " on " + report["device"])
    np.savez_compressed(out_dir / "blackwell_golden.npz", **store)
    (out_dir / "blackwell_reference_report.json").write_text(json.dumps(report, indent=1))
    print("wrote", out_dir / "blackwell_golden.npz", flush=True)


EXT_CASES = (("small", 100, 256, 512), ("w4a8_gate_up", 816, 16384, 2048), ("producer_kv", 816, 256, 2048))


def main_ext(out_dir):
    """Second fixture file, `blackwell_golden_ext.npz`: the reference's W4A8-MX packers and GEMM
    (`robotics_cutlass_fp4_mx`), its FP8 producer GEMM, and its SwiGLU -> NVFP4 -> GEMM chain in both
    gate/up layouts, beside this library's results on the same inputs."""
    from oracle import ref_kernels as RK
    from rk_b200 import fp4_linear as P4
    from rk_b200 import fp4_mx_linear as PM
    from rk_b200 import fp8_linear as P8

    dev = torch.device("cuda:0")
    torch.cuda.set_device(0)
    store, report = {}, {"device": torch.cuda.get_device_name(0), "cases": {}, "timing_us": {}}
    mx, why_mx = RK.load("fp4_mx")
    f8, why_f8 = RK.load("fp8")
    f4, why_f4 = RK.load("fp4")
    report["extensions"] = {"fp4_mx": why_mx or "loaded", "fp8": why_f8 or "loaded", "fp4": why_f4 or "loaded"}
    for name, m, n, k in EXT_CASES:
        full = name == "small"
        x, w, bias = (t.to(dev) for t in case_inputs(name, m, n, k))
        entry = report["cases"].setdefault(name, {"m": m, "n": n, "k": k})
        timing = report["timing_us"].setdefault(name, {})
        if mx is not None and name != "producer_kv":
            ra, rfa = mx.pack_mxfp8_activation(x)
            rb, rfb, meta = mx.pack_mxfp4_weight(w, "linear", name)
            oa, ofa = PM.pack_mxfp8_activation(x)
            ob, ofb = PM.pack_mxfp4_weight(w)
            entry["w4a8"] = {
                "a_codes_differ": store_array(store, f"{name}_w4a8_a_codes", ra, oa, full),
                "a_sf_differ": store_array(store, f"{name}_w4a8_a_sf", rfa.reshape(-1), ofa, full),
                "w_codes_differ": store_array(store, f"{name}_w4a8_w_codes", rb, ob, full),
                "w_sf_differ": store_array(store, f"{name}_w4a8_w_sf", rfb.reshape(-1), ofb, full)}
            ref = mx.linear_w4a8_packed(ra, rfa, rb, rfb, meta, bias)
            mine = PM.linear_w4a8_packed(ra.view(torch.float8_e4m3fn), rfa.reshape(-1).contiguous(), rb,
                                         rfb.reshape(-1).contiguous(), bias)
            entry["w4a8"]["gemm"] = compare_out(ref, mine)
            store[f"{name}_w4a8_out_sample"] = out_sample(ref)
            store[f"{name}_w4a8_out_ours_sample"] = out_sample(mine)
            if full:
                store[f"{name}_w4a8_out"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
            timing["w4a8_ref"] = time_us(lambda: mx.linear_w4a8_packed(ra, rfa, rb, rfb, meta, bias))
            rfa1, rfb1 = rfa.reshape(-1).contiguous(), rfb.reshape(-1).contiguous()
            ra8 = ra.view(torch.float8_e4m3fn)
            timing["w4a8_ours"] = time_us(lambda: PM.linear_w4a8_packed(ra8, rfa1, rb, rfb1, bias))
            print(name, "w4a8", entry["w4a8"], timing, flush=True)
        if f8 is not None and name != "w4a8_gate_up":
            wq, wscale = f8.quantize_bf16(w)
            ref = f8.linear_forward_producer(x, wq, wscale, bias)
            mine = P8.linear_forward_producer(x, wq, wscale.reshape(1), bias)
            entry["fp8_producer"] = compare_out(ref, mine)
            store[f"{name}_fp8prod_w_scale"] = wscale.reshape(1).cpu().numpy()
            store[f"{name}_fp8prod_w_codes_sha"] = np.array(sha(wq.view(torch.uint8).cpu().numpy()))
            store[f"{name}_fp8prod_out_sample"] = out_sample(ref)
            store[f"{name}_fp8prod_out_ours_sample"] = out_sample(mine)
            if full:
                store[f"{name}_fp8prod_w_codes"] = wq.view(torch.uint8).cpu().numpy()
                store[f"{name}_fp8prod_out"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
            timing["fp8_producer_ref"] = time_us(lambda: f8.linear_forward_producer(x, wq, wscale, bias))
            ws1 = wscale.reshape(1)
            timing["fp8_producer_ours"] = time_us(lambda: P8.linear_forward_producer(x, wq, ws1, bias))
            print(name, "fp8 producer", entry["fp8_producer"], timing, flush=True)
        del x, w
        torch.cuda.empty_cache()

    # SwiGLU chains (small): gate_up [100, 2 * 768] -> down projection [256, 768]
    x, res, weight, gate_up, inter = (t.to(dev) if torch.is_tensor(t) else t for t in producer_inputs())
    gen = torch.Generator().manual_seed(78)
    wd = (torch.randn(256, inter, generator=gen) * 0.02).to(torch.bfloat16).to(dev)
    lin = torch.nn.Linear(inter, 256, bias=False, device=dev, dtype=torch.bfloat16)
    with torch.no_grad():
        lin.weight.copy_(wd)
    if f4 is not None:
        rb, rfb, meta = f4.pack_linear_weight_gemm_bf16(wd, "linear", "down")
        layer = P4.Fp4CutlassLinear.from_linear(lin, "linear", "down")
        for interleaved in (False, True):
            ref = f4.linear_forward_swiglu_gemm_bf16(gate_up, inter, rb, rfb, meta, None, "linear", "down", interleaved)
            mine = layer.forward_swiglu(gate_up, inter, interleaved)
            report["cases"][f"nvfp4_swiglu_chain_{int(interleaved)}"] = compare_out(ref, mine)
            store[f"swiglu_nvfp4_out_{int(interleaved)}"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
    if mx is not None:
        rb, rfb, meta = mx.pack_mxfp4_weight(wd, "linear", "down")
        layer = PM.Fp4MxLinear.from_linear(lin, "linear", "down")
        for interleaved in (False, True):
            rq, rsf = mx.pack_swiglu_mxfp8(gate_up, inter, interleaved)
            oq, osf = PM.pack_swiglu_mxfp8(gate_up, inter, interleaved)
            tag = f"swiglu_mxfp8_{int(interleaved)}"
            report["cases"][tag] = {"codes_differ": store_array(store, tag + "_codes", rq, oq, True),
                                    "sf_differ": store_array(store, tag + "_sf", rsf.reshape(-1), osf, True)}
            ref = mx.linear_w4a8_packed(rq, rsf, rb, rfb, meta, None)
            mine = layer.forward_swiglu(gate_up, inter, interleaved)
            report["cases"][tag]["chain"] = compare_out(ref, mine)
            store[tag + "_out"] = ref.view(torch.int16).cpu().numpy().view(np.uint16)
    print(json.dumps({k: v for k, v in report["cases"].items() if "swiglu" in k}), flush=True)
    out_dir = Path(out_dir)
    out_dir.mkdir(parents=True, exist_ok=True)
    store["generated"] = np.array(time.strftime("%Y-%m-%d") + " on " + report["device"])
    np.savez_compressed(out_dir / "blackwell_golden_ext.npz", **store)
    (out_dir / "blackwell_reference_report_ext.json").write_text(json.dumps(report, indent=1))
    print("wrote", out_dir / "blackwell_golden_ext.npz", flush=True)


SILU_CASES = (("small", 100, 768), ("mlp", 816, 4096))  # (name, rows, intermediate size)


def silu_inputs(name, rows, inter):
    gen = torch.Generator().manual_seed(2000 + sum(ord(c) for c in name))
    gate_up = (torch.randn(rows, 2 * inter, generator=gen) * 2.0).to(torch.bfloat16)
    if name == "small":
        gate_up[3, 5] = float("inf")  # a non-finite block gets the scale byte 255
        gate_up[4, :32] = 0           # an all-zero block
    return gate_up


def main_silu(out_dir):
    """Third fixture file, `blackwell_golden_silu.npz`: the reference's table-SiLU SwiGLU producer for
    MXFP8 (`robotics_mxfp8_swiglu::silu_mul_pack`), with the table it was given, beside this library's."""
    from oracle import ref_kernels as RK
    from rk_b200 import mxfp8_swiglu as MS

    dev = torch.device("cuda:0")
    torch.cuda.set_device(0)
    ns, why = RK.load("mxfp8_swiglu")
    if ns is None:
        raise SystemExit(f"reference extension unavailable: {why}")
    store, report = {}, {"device": torch.cuda.get_device_name(0), "cases": {}}
    table = MS.make_bf16_silu_table(dev)
    store["silu_table_bits"] = table.view(torch.int16).cpu().numpy().view(np.uint16)
    for name, rows, inter in SILU_CASES:
        gate_up = silu_inputs(name, rows, inter).to(dev)
        rq, rsf = ns.silu_mul_pack(gate_up, inter, table)
        oq, osf = MS.silu_mul_pack_mxfp8(gate_up, inter, table)
        tag = "silu_" + name
        report["cases"][tag] = {
            "codes_differ": store_array(store, tag + "_codes", rq.view(torch.uint8), oq.view(torch.uint8), name == "small"),
            "sf_differ": store_array(store, tag + "_sf", rsf.reshape(-1), osf, name == "small")}
    print(json.dumps(report["cases"]), flush=True)
    out_dir = Path(out_dir)
    out_dir.mkdir(parents=True, exist_ok=True)
    store["generated"] = np.array(time.strftime("%Y-%m-%d") + " on " + report["device"])
    np.savez_compressed(out_dir / "blackwell_golden_silu.npz", **store)
    (out_dir / "blackwell_reference_report_silu.json").write_text(json.dumps(report, indent=1))
    print("wrote", out_dir / "blackwell_golden_silu.npz", flush=True)


if __name__ == "__main__":
    args = [a for a in sys.argv[1:] if not a.startswith("--")]
    target = args[0] if args else "golden_out"
    if "--ext" in sys.argv:
        main_ext(target)
    elif "--silu" in sys.argv:
        main_silu(target)
    else:
        main(target)
