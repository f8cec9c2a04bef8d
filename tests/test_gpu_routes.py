"""Kernels that a rule on sizes picks, at the sizes where the rule changes and where their tiles and pieces end."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import kipizen_ref
import mufevik_ref as ref
from oracle import ref as oracle
from onyxia_b200 import backend as be
from onyxia_b200 import ir, kipizen, llm, lovuzen, models
from onyxia_b200.ir import HostTensor
from gpu_util import cuda_backend, differential
from lovuzen_util import to_bf16
from test_gpu_kipizen import Attention, Experts, piece, row_err
import test_gpu_lovuzen
import test_gpu_mufevik
from test_gpu_lovuzen import act, attention_want, rel_err, run_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 8, 9, 32, 33, 65])
def test_f32_products_with_long_sums(rows):
    """Weight rows shared by 1 … 8 warps, four and eight of them per warp; tiles cut along k; a second operand that begins inside a step.
    A sum of k products in pieces is off by at most about (k / 32 + 10) · 2^-24 of the sum of magnitudes; 2e-6 holds with room for k ≤ 7000."""
    r = np.random.default_rng(rows)
    for k, k1, n in ((4100, 0, 52), (6912, 260, 1154), (1152, 0, 2370), (132, 0, 20001)):
        x, w = r.standard_normal((rows, k)).astype(np.float32), r.standard_normal((n, k)).astype(np.float32)
        want, more = x.astype(np.float64) @ w.T.astype(np.float64), {}
        if k1:
            more = {"x1": r.standard_normal((rows, k1)).astype(np.float32), "w1": r.standard_normal((n, k1)).astype(np.float32)}
            want = want + more["x1"].astype(np.float64) @ more["w1"].T.astype(np.float64)
        bias = r.standard_normal(n).astype(np.float32)
        assert rel_err(run_linear(ir.F32, x, w, bias=bias, **more), want + bias) < 2e-6, (k, n)


@pytest.mark.parametrize("dtype,d,seq", [(ir.F16, 64, 1), (ir.F16, 128, 1), (ir.F16, 256, 1), (ir.F32, 64, 1), (ir.F16, 64, 3), (ir.F32, 32, 5), (ir.F16, 128, 20)])
def test_caches_are_copied_into_a_new_buffer(dtype, d, seq):
    """A step on caches that it cannot append to: the past arrives bit for bit (several CTAs per head, the last one short), what lies behind a
    ragged row is zero, and the results are those of the decomposition within the tests' tolerances for these types."""
    batch, past = 3, 517
    module, feed = models.build_gqa(batch, 4, 2, d, past, seq, dtype, -1, True, seed=d + seq)
    valid = [past, 130, 0]
    feed["seqlens_k"] = HostTensor.from_numpy(np.array([v + seq - 1 for v in valid], np.int32))
    tol = dict(atol=4e-3, rtol=4e-3) if dtype == ir.F16 else dict(atol=2e-4, rtol=1e-3)
    got = {n: t.numpy() for n, t in differential(module, feed, **tol)[0]}
    for name in ("key", "value"):
        for b, v in enumerate(valid):
            assert np.array_equal(got["present_" + name][b, :, :v], feed["past_" + name].numpy()[b, :, :v])
            assert not got["present_" + name][b, :, v + seq:].any()


def widened(packed, scales, n, nb, zero=8.0):
    """The weights as the decomposition rounds them: (q − zero) · scale in the scales' type."""
    q = np.stack([packed & 15, packed >> 4], 1).reshape(n, nb, 32).astype(np.float64)
    return ((q - zero) * scales.astype(np.float64).reshape(n, nb, 1)).astype(scales.dtype).astype(np.float64).reshape(n, nb * 32)


@pytest.mark.parametrize("m,k,n", [(257, 1152, 1536), (300, 1000, 200), (513, 136, 4104), (384, 6912, 4760), (300, 1152, 29300)])
def test_many_rows_against_weights_widened_once(m, k, n):
    """Tiles that end inside a tile, k that ends inside a block and inside a step, one and two panels of weights, whole k and pieces of it.
    After one rounding to f16 nearly all outputs equal the f64 sum's (the bound of the other kernel's test), none is further than an ulp of
    the largest away."""
    module, act = models.build_matmul_nbits(m, k, n, act_dtype=ir.F16, seed=m)
    cfg = models.DecoderConfig("nbits", 0, 0, 0, 0, 0, 0, 0)
    packed, scales, _ = models.nbits_arrays(cfg, m, f"w{k}x{n}", k, n)
    want = (act.numpy().astype(np.float64) @ widened(packed, scales, n, (k + 31) // 32)[:, :k].T).astype(np.float16)
    got = be.run_once(cuda_backend(), module, {"a": act})[0][1].numpy()
    assert (got != want).mean() <= 0.01
    assert np.abs(got.astype(np.float32) - want.astype(np.float32)).max() <= 2.0 ** -10 * np.abs(want.astype(np.float32)).max()


@pytest.mark.parametrize("act_dtype", [ir.F32, ir.F16])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 9, 17])
def test_generic_int4_products(act_dtype, m):
    """Every number of activation rows per pass; 1, 2, 4 and 8 warps per unit of weight rows; k that ends inside a lane's eight. f32: sums of k
    products in 32 chains per warp are off by less than (k / 256 + 8) · 2^-24 of the sum of magnitudes."""
    r = np.random.default_rng(m)
    for k, n in ((512, 10), (2048, 515), (50, 7), (6912, 36), (1000, 2500)):
        nb = (k + 31) // 32
        packed, scales = r.integers(0, 256, n * nb * 16, dtype=np.uint8), r.uniform(0.005, 0.02, n * nb).astype(np.float32)
        a = r.standard_normal((m, k)).astype(np.float32 if act_dtype == ir.F32 else np.float16)
        b = ir.GraphBuilder()
        x = b.input("a", act_dtype, [m, k])
        ins = [x, b.constant(HostTensor(ir.U4, [n, nb, 32], packed)), b.constant(HostTensor.from_numpy(scales))]
        b.output("y", b.composite("com.microsoft.MatMulNBits", {"K": k, "N": n, "bits": 4, "block_size": 32}, ins, [(act_dtype, [m, n])])[0])
        got = be.run_once(cuda_backend(), b.finish(), {"a": HostTensor.from_numpy(a)})[0][1].numpy()
        w = widened(packed, scales, n, nb)[:, :k]
        if act_dtype == ir.F16:
            w = w.astype(np.float16).astype(np.float64)
        assert rel_err(got.astype(np.float64), a.astype(np.float64) @ w.T) < (1e-6 if act_dtype == ir.F32 else 4e-4), (k, n)


@pytest.mark.parametrize("rows", [1, 3, 8, 9, 17, 32])
def test_bf16_products_of_few_rows(rows):
    """Matrices below and above the line to linear_flow: several tiles per CTA, k that ends inside a chunk and with some warps only, a second
    operand that begins inside the warps' turn, rings that wrap. Inputs are on the bf16 grid and products exact: f32 sums of k products are off
    by less than 2e-6 of the result's rms."""
    r = np.random.default_rng(rows)
    for k, k1, n in ((4608, 0, 1152), (2056, 136, 5003), (1152, 0, 15000), (40, 0, 260000), (1096, 0, 2400)):
        x, w, more = to_bf16(r.standard_normal((rows, k))), to_bf16(r.standard_normal((n, k))), {}
        want = x.astype(np.float64) @ w.T.astype(np.float64)
        if k1:
            more = {"x1": to_bf16(r.standard_normal((rows, k1))), "w1": to_bf16(r.standard_normal((n, k1)))}
            want = want + more["x1"].astype(np.float64) @ more["w1"].T.astype(np.float64)
        assert rel_err(run_linear(ir.BF16, x, w, **more), want) < 2e-6, (k, n)
    x, w = to_bf16(r.standard_normal((rows, 2304))), to_bf16(r.standard_normal((4402, 2304)) / 48)
    z = x.astype(np.float64) @ w.T.astype(np.float64)
    g, u = np.minimum(z[:, ::2], 1.5), np.clip(z[:, 1::2], -1.5, 1.5)
    assert rel_err(run_linear(ir.BF16, x, w, glu=(1.7, 1.5, 1.0)), g / (1 + np.exp(-1.7 * g)) * (u + 1)) < 3e-6


@pytest.mark.parametrize("rows", [1, 7, 8, 9])
def test_norms_in_front_of_a_large_matrix(rows):
    """Every norm that runs as the prologue, in front of 20 MB and more. Tolerances as for small matrices: the norm's operand is rounded to bf16."""
    r = np.random.default_rng(rows)
    eps, n, of = 1e-3, 19999, HostTensor.from_numpy
    for kind, width in (("residual", 520), ("streams", 528), ("groups", 544)):
        y, w, m = to_bf16(0.02 * r.standard_normal((rows, width))).astype(np.float32), to_bf16(r.standard_normal(width)), to_bf16(r.standard_normal((n, width)))
        S = 3 if kind == "streams" else 1
        b, feed = ir.GraphBuilder(), {"y": of(y)}
        ins, y64 = [b.input("y", ir.F32, [rows, width])], y.astype(np.float64)
        if kind == "groups":
            w, gate = np.tile(w[:136], 4), to_bf16(r.standard_normal((rows, width)))
            ins += [b.constant(of(w)), b.input("gate", ir.BF16, [rows, width])]
            feed["gate"], attrs = act(gate, ir.BF16), {"norm_groups": 4, "gate": 1, "gate_offset": 0}
            want = ref.rms_norm(y64.reshape(rows, 4, 136), w[:136], eps).reshape(rows, width) * gate
        else:
            res = (0.1 * r.standard_normal((rows, S, width))).astype(np.float32)
            ins += [b.constant(of(w)), b.input("res", ir.F32, [rows, S * width])]
            feed["res"], attrs = of(res.reshape(rows, -1)), {"residual": 1}
            want = ref.rms_norm(y64, w, eps) + res[:, 0]
            if S > 1:
                mix, out, take = r.standard_normal((S, S)), r.standard_normal(S), r.standard_normal(S)
                ins.append(b.constant(of(np.concatenate([mix.reshape(-1), out, take]).astype(np.float32))))
                attrs.update(pre=1, streams=S)
                new = out[None, :, None] * y64[:, None] + np.einsum("st,rsw->rtw", mix, res.astype(np.float64))
                want = ref.rms_norm(np.einsum("t,rtw->rw", take, new), w, eps)
        b.output("out", b.composite("onyxia.Linear", dict(attrs, epsilon=eps, norm=1, stream=0), ins + [b.constant(act(m, ir.BF16))], [(ir.F32, [rows, n])])[0])
        got = be.run_once(cuda_backend(), b.finish(), feed)[0][1].numpy()
        assert rel_err(got, want @ m.T.astype(np.float64)) < 6e-3, kind


@pytest.mark.parametrize("rows", [40, 300, 1100])
def test_bf16_products_in_persistent_tiles(rows):
    """More tiles than resident CTAs, the last round short; tiles that end inside a tile in both directions; plain, gated, with a function."""
    r = np.random.default_rng(rows)
    for k, n in ((136, 20010), (520, 9000)):
        x, w = to_bf16(r.standard_normal((rows, k))), to_bf16(r.standard_normal((n, k)) / np.sqrt(k))
        z = x.astype(np.float64) @ w.T.astype(np.float64)
        assert rel_err(run_linear(ir.BF16, x, w), z) < 2e-6
        g, u = np.minimum(z[:, ::2], 2.0), np.clip(z[:, 1::2], -2.0, 2.0)
        assert rel_err(run_linear(ir.BF16, x, w, glu=(1.7, 2.0, 1.0)), g / (1 + np.exp(-1.7 * g)) * (u + 1)) < 3e-6


@pytest.mark.parametrize("n", [1, 8, 9, 32, 70, 600])
def test_experts_with_long_products(n):
    """Long sums of both products, pieces of the second one over clusters; grouped tiles of many experts. `check` compares with
    the plain implementation at the tolerance of its own tests."""
    m = Experts("bf16", 1160, 12, 3, 840)
    m.check(m.rows(n))


def test_gelu_of_every_half():
    """All 65 536 values, many times over, alone and times another: the table's bits are those of the element-wise kernel that small tensors take."""
    bits = np.arange(65536, dtype=np.uint16).view(np.float16)
    for form in ("tanh", "none"):
        outs = []
        for copies in (1, 17):
            x = np.tile(bits, copies)
            m = (0.5 + np.arange(x.size) % 7).astype(np.float16)
            b = ir.GraphBuilder()
            xi, mi = b.input("x", ir.F16, [x.size]), b.input("m", ir.F16, [x.size])
            g = b.composite("Gelu", {"approximate": form}, [xi], [(ir.F16, [x.size])])[0]
            h = b.composite("Gelu", {"approximate": form}, [xi], [(ir.F16, [x.size])])[0]
            b.output("g", g)
            b.output("p", b.mul(h, mi))
            got = be.run_once(cuda_backend(), b.finish(), {"x": HostTensor.from_numpy(x), "m": HostTensor.from_numpy(m)})
            outs.append([v.numpy()[:65536] for _, v in got])
        assert np.array_equal(outs[0][0], outs[1][0], equal_nan=True) and np.array_equal(outs[0][1], outs[1][1], equal_nan=True)


def test_gelu_beside_another_streams_capture():
    """The table's first use in a process leaves a graph that is being recorded on another stream as it is."""
    code = """if True:
        import numpy as np
        import torch
        from onyxia_b200 import backend as be, ir
        from onyxia_b200.ir import HostTensor
        n = 1 << 20
        b = ir.GraphBuilder()
        b.output("y", b.composite("Gelu", {"approximate": "tanh"}, [b.input("x", ir.F16, [n])], [(ir.F16, [n])])[0])
        s = be.CudaBackend((0,)).prepare(b.finish())
        x = s.upload(HostTensor.from_numpy(np.ones(n, np.float16)))
        t, graph = torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            graph.capture_begin(capture_error_mode="relaxed")
            t += 1
            s.run({"x": x})
            t += 1
            graph.capture_end()
        graph.replay()
        torch.cuda.synchronize()
        assert t.tolist() == [2.0] * 4
    """
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("heads,kv,d,past,seq,window", [(4, 1, 256, 0, 100, -1), (8, 2, 64, 300, 40, 70), (3, 3, 128, 50, 33, -1), (6, 2, 128, 0, 700, 129),
                                                        (2, 1, 64, 1, 16, 0), (8, 2, 64, 300, 40, -1), (6, 2, 128, 0, 700, 300), (4, 1, 256, 0, 200, -1),
                                                        (2, 1, 64, 300, 16, 260)])
def test_prefill_attention_with_kept_scores(heads, kv, d, past, seq, window):
    """Pairs of heads and single ones, windows shorter and longer than a block, ranges that end inside a block, a query tile that is not full;
    the bounds are those of the kernel's own tests (every rounding of the decomposition is repeated, sums differ in the last bits)."""
    module, feed = models.build_gqa(2, heads, kv, d, past, seq, ir.F16, window, True, seed=seq)
    got, want = differential(module, feed, atol=4e-3, rtol=4e-3)
    g, w = got[0][1].numpy(), want[0][1].numpy()
    assert (g != w).mean() <= 0.15


@pytest.mark.parametrize("rows,k,k1,n", [(1100, 2056, 0, 9000), (700, 1032, 1032, 12000), (2048, 1152, 0, 4610)])
def test_bf16_products_of_several_rounds_per_cta(rows, k, k1, n):
    """More tiles than SMs: tiles that end early in both directions, several rounds per CTA, a second operand, rings that wrap."""
    r = np.random.default_rng(rows)
    x, w, more = to_bf16(r.standard_normal((rows, k))), to_bf16(r.standard_normal((n, k)) / np.sqrt(k)), {}
    z = x.astype(np.float64) @ w.T.astype(np.float64)
    if k1:
        more = {"x1": to_bf16(r.standard_normal((rows, k1))), "w1": to_bf16(r.standard_normal((n, k1)) / np.sqrt(k1))}
        z = z + more["x1"].astype(np.float64) @ more["w1"].T.astype(np.float64)
    bias = to_bf16(r.standard_normal(n))
    assert rel_err(run_linear(ir.BF16, x, w, bias=bias, **more), z + bias) < 2e-6
    if not k1:
        z = z + bias
        g, u = np.minimum(z[:, ::2], 2.0), np.clip(z[:, 1::2], -2.0, 2.0)
        assert rel_err(run_linear(ir.BF16, x, w, bias=bias, glu=(1.7, 2.0, 1.0)), g / (1 + np.exp(-1.7 * g)) * (u + 1)) < 3e-6


@pytest.mark.parametrize("rows,k,k1,n,out", [(257, 1160, 0, 13830, ir.F32), (700, 72, 0, 9001, ir.BF16), (1999, 1152, 136, 2370, ir.BF16), (2048, 16, 0, 2560, ir.F32), (3001, 520, 0, 1536, ir.BF16)])
def test_bf16_products_by_pairs_of_ctas(rows, k, k1, n, out):
    """Tiles that end inside a CTA's weight rows or in the first CTA of a pair, odd columns, last tiles of few rows, a k below one step, a second operand inside the ring,
    tiles of sizes between the powers of two, several rounds. Products are exact; f32 sums as above, a bf16 result is off by half a unit of eight digits."""
    r = np.random.default_rng(rows)
    x, w, more = to_bf16(r.standard_normal((rows, k))), to_bf16(r.standard_normal((n, k)) / np.sqrt(k)), {}
    z = x.astype(np.float64) @ w.T.astype(np.float64)
    if k1:
        more = {"x1": to_bf16(r.standard_normal((rows, k1))), "w1": to_bf16(r.standard_normal((n, k1)) / np.sqrt(k))}
        z = z + more["x1"].astype(np.float64) @ more["w1"].T.astype(np.float64)
    b = ir.GraphBuilder()
    b.output("y", b.composite("onyxia.Linear", {}, [b.input("x", ir.BF16, [rows, k]), b.constant(act(w, ir.BF16))], [(out, [rows, n])])[0])
    assert kernels_of(b.finish(), {"x": act(x, ir.BF16)}) == {"linear_pair"}
    bias = to_bf16(r.standard_normal(n))
    assert rel_err(run_linear(ir.BF16, x, w, bias=bias, out_dtype=out, **more).astype(np.float64), z + bias) < (2e-6 if out == ir.F32 else 2.0 ** -9)
    if n % 2 == 0 and not k1:
        g, u = np.minimum(z[:, ::2], 2.0), np.clip(z[:, 1::2], -2.0, 2.0)
        assert rel_err(run_linear(ir.BF16, x, w, glu=(1.7, 2.0, 1.0), out_dtype=out).astype(np.float64), g / (1 + np.exp(-1.7 * g)) * (u + 1)) < (3e-6 if out == ir.F32 else 2.0 ** -9)
    b, z = ir.GraphBuilder(), x.astype(np.float64) @ w.T.astype(np.float64)
    attrs = {"act": "silu", "act_rest": "softplus", "act_split": n // 3, "act_end": n - 5}
    b.output("y", b.composite("onyxia.Linear", attrs, [b.input("x", ir.BF16, [rows, k]), b.constant(act(w, ir.BF16))], [(out, [rows, n])])[0])
    z[:, :n // 3] /= 1 + np.exp(-z[:, :n // 3])
    z[:, n // 3:n - 5] = np.log1p(np.exp(z[:, n // 3:n - 5]))
    got = be.run_once(cuda_backend(), b.finish(), {"x": act(x, ir.BF16)})[0][1].numpy().astype(np.float64)
    assert rel_err(got, z) < (3e-6 if out == ir.F32 else 2.0 ** -9)


@pytest.mark.parametrize("n,experts,top,width,ff", [(700, 3, 2, 1160, 1100), (1500, 5, 1, 1160, 1096), (600, 4, 4, 264, 1700), (4000, 40, 2, 264, 1100)])
def test_experts_by_pairs_of_ctas(n, experts, top, width, ff):
    """Groups of a few parts each, some of hardly a row more than a tile, more groups than a warp's search takes at once."""
    m = Experts("bf16", width, experts, top, ff)
    h = m.rows(n)
    m.check(h)
    m.s.enable_profiling(True)
    m.check(h)
    assert "grouped_pair" in {kernel for kernel, _, _ in m.s.take_timings()}


@pytest.mark.parametrize("d,past,seq,window", [(64, 240, 33, -1), (128, 100, 300, 250), (256, 300, 20, 150)])
def test_kept_scores_with_values_that_are_not_finite(d, past, seq, window):
    """Rows whose visible scores are NaN, all minus infinity, or infinite in part, and a NaN among the keys: kept scores (two heads per key head) give
    what the kernel that walks the keys three times gives for the same heads with a key head each, bit for bit in the other rows too."""
    pairs, feed = models.build_gqa(2, 4, 2, d, past, seq, ir.F16, window, False, seed=d)
    single, _ = models.build_gqa(2, 4, 4, d, past, seq, ir.F16, window, False, seed=d)
    x = {n: t.numpy().copy() for n, t in feed.items()}
    q, k = x["q"].reshape(2, seq, 4, d), x["k"].reshape(2, seq, 2, d)
    k[..., 0], x["past_key"][..., 0] = 100, 100
    q[..., 0] = 0
    q[0, 3, 1] = np.nan           # every score of the row
    q[0, 5, 2, 0] = -60000        # every score overflows to minus infinity
    q[1, 7, 0, 1] = 60000         # scores of both signs
    k[1, 9, 1, 2] = np.nan        # one key
    feed = {n: HostTensor.from_numpy(v) for n, v in x.items()}
    got = be.run_once(cuda_backend(), pairs, feed)[0][1].numpy().reshape(2, seq, 4, d)
    for n in ("k", "v"):
        feed[n] = HostTensor.from_numpy(np.repeat(x[n].reshape(2, seq, 2, d), 2, axis=2).reshape(2, seq, 4 * d))
    for n in ("past_key", "past_value"):
        feed[n] = HostTensor.from_numpy(np.repeat(x[n], 2, axis=1))
    want = be.run_once(cuda_backend(), single, feed)[0][1].numpy().reshape(2, seq, 4, d)
    assert np.isnan(got[0, 3, 1]).all() and np.isnan(got[0, 5, 2]).all() and np.isnan(got[1, 9, 2]).all()
    assert np.array_equal(got, want, equal_nan=True) and np.isfinite(got[:, :3]).all()


def test_windows_up_to_the_largest_number():
    """A window beyond all positions sees what no window sees, up to the type's largest value."""
    feeds = [models.build_gqa(1, 4, 2, 64, 300, 30, ir.F16, w, True, seed=1) for w in (-1, 330, 2 ** 63 - 17, 2 ** 63 - 16, 2 ** 63 - 1)]
    want, *got = [be.run_once(cuda_backend(), m, f)[0][1].numpy() for m, f in feeds]
    assert all(np.array_equal(g, want) for g in got)


@pytest.mark.parametrize("d", [64, 128, 256])
def test_single_tokens_behind_a_copied_cache_keep_their_sums_in_64_bits(d):
    """The outputs are the oracle's, whose sums are in f64, bit for bit: sums of these lengths in f64 round to other f16 values only at ties."""
    module, feed = models.build_gqa(3, 8, 2, d, 900, 1, ir.F16, -1, True, seed=d)
    got, want = differential(module, feed, atol=4e-3, rtol=4e-3)
    assert (got[0][1].numpy() != want[0][1].numpy()).mean() <= 2e-4


def test_plans_of_changing_sizes_share_one():
    """Sizes that come twice each, as the rows of a serving batch do: one plan is patched for all of them, and its memory is that of the largest."""
    k, n, nb = 1024, 512, 32
    r = np.random.default_rng(0)
    b = ir.GraphBuilder()
    rows = b.sym("rows")
    ins = [b.input("a", ir.F16, [rows, k]), b.constant(HostTensor(ir.U4, [n, nb, 32], r.integers(0, 256, n * nb * 16, dtype=np.uint8))),
           b.constant(HostTensor.from_numpy(r.uniform(0.005, 0.02, n * nb).astype(np.float16)))]
    y = b.composite("com.microsoft.MatMulNBits", {"K": k, "N": n, "bits": 4, "block_size": 32}, ins, [(ir.F16, [rows, n])])[0]
    b.output("y", b.composite("Gelu", {"approximate": "tanh"}, [y], [(ir.F16, [rows, n])])[0])
    s = cuda_backend().prepare(b.finish())
    held = []
    for m in (600, 590, 400, 64, 300, 33, 500, 20, 280, 599):
        a = s.upload(HostTensor.from_numpy(r.standard_normal((m, k)).astype(np.float16)))
        for _ in range(2):
            s.run({"a": a})
        s.wait_idle()
        del a
        held.append(s.resident_bytes())
    stats = s.plan_stats()
    assert stats["built"] == 1 and stats["updated"] == 9
    assert max(held) <= held[0]


def kernels_of(module, feed):
    """Names of the kernels that a run launches."""
    s = cuda_backend().prepare(module)
    s.enable_profiling(True)
    s.run({n: s.upload(t) for n, t in feed.items()})
    return {kernel for kernel, _, _ in s.take_timings()}


@pytest.mark.parametrize("m,k,n,wide", [(256, 512, 64, False), (257, 128, 64, True), (257, 1152, 6912, True), (257, 4096, 1024, True), (512, 4096, 1024, False),
                                        (257, 5376, 2048, True), (512, 5376, 2048, False), (1024, 5376, 2048, True), (512, 8192, 2048, False)])
def test_where_int4_weights_are_widened_once(m, k, n, wide):
    module, act = models.build_matmul_nbits(m, k, n, act_dtype=ir.F16, seed=m)
    names = kernels_of(module, {"a": act})
    assert ("nbits_gemm_wide" in names) == wide and ("nbits_gemm_tc" in names) != wide


@pytest.mark.parametrize("m,parts,k,n,zp", [(400, 2, 1000, 200, True), (512, 2, 1152, 1536, False), (400, 2, 136, 4104, True), (384, 2, 1152, 29300, True),
                                            (1024, 4, 4096, 2064, False), (1024, 5, 6912, 1152, True)])
def test_weights_widened_once_give_the_bits_of_the_passes(m, parts, k, n, zp):
    """The same rows in pieces of 129 to 256, which take the passes: pieces of k and whole k, k that ends inside a block, two panels, zero points."""
    module, act = models.build_matmul_nbits(m, k, n, act_dtype=ir.F16, seed=n, with_zp=zp)
    got = be.run_once(cuda_backend(), module, {"a": act})[0][1].numpy()
    for rows in np.array_split(np.arange(m), parts):
        part, _ = models.build_matmul_nbits(len(rows), k, n, act_dtype=ir.F16, seed=n, with_zp=zp)
        feed = {"a": HostTensor.from_numpy(act.numpy()[rows].copy())}
        assert np.array_equal(got[rows], be.run_once(cuda_backend(), part, feed)[0][1].numpy())


@pytest.mark.parametrize("dtype,rows,k,n,kernel", [(ir.BF16, 8, 9216, 1100, "linear_flow"), (ir.BF16, 16, 8192, 1200, "linear_flow"), (ir.BF16, 9, 8200, 1200, "linear_stream"),
                                                   (ir.BF16, 17, 8200, 1200, "linear_flow"), (ir.BF16, 32, 12288, 800, "linear_flow"), (ir.BF16, 32, 12296, 800, "linear_stream")])
def test_where_few_rows_take_the_ring(dtype, rows, k, n, kernel):
    """The line itself, and the product on both sides of it: f32 sums of exact products, as in the test above."""
    r = np.random.default_rng(k)
    x, w = to_bf16(r.standard_normal((rows, k))), to_bf16(r.standard_normal((n, k)))
    b = ir.GraphBuilder()
    b.output("y", b.composite("onyxia.Linear", {}, [b.input("x", dtype, [rows, k]), b.constant(act(w, dtype))], [(ir.F32, [rows, n])])[0])
    module, feed = b.finish(), {"x": act(x, dtype)}
    assert kernels_of(module.clone(), feed) == {kernel}
    assert rel_err(be.run_once(cuda_backend(), module, feed)[0][1].numpy(), x.astype(np.float64) @ w.T.astype(np.float64)) < 2e-6


@pytest.mark.parametrize("rows,k,kernel", [(1, 16, "linear_simt"), (40, 64, "linear_simt"), (33, 188, "linear_simt"), (2, 192, "linear_f32"), (40, 192, "linear_f32"),
                                           (8, 508, "linear_f32"), (8, 512, "linear_rows_f32")])
def test_where_f32_products_take_register_tiles(rows, k, kernel):
    """The line itself, and sums of k products of f32 on both sides of it: off by less than (k + 2) · 2^-24 of the sum of magnitudes."""
    r = np.random.default_rng(k)
    x, w = r.standard_normal((rows, k)).astype(np.float32), r.standard_normal((70, k)).astype(np.float32)
    b = ir.GraphBuilder()
    b.output("y", b.composite("onyxia.Linear", {}, [b.input("x", ir.F32, [rows, k]), b.constant(HostTensor.from_numpy(w))], [(ir.F32, [rows, 70])])[0])
    module, feed = b.finish(), {"x": HostTensor.from_numpy(x)}
    assert kernels_of(module.clone(), feed) - {"linear_reduce"} == {kernel}
    assert rel_err(be.run_once(cuda_backend(), module, feed)[0][1].numpy(), x.astype(np.float64) @ w.T.astype(np.float64)) < 2e-6


@pytest.mark.parametrize("heads,kv,d,seq,window,batch,kept", [(4, 1, 256, 159, -1, 1, False), (4, 1, 256, 160, -1, 1, True), (8, 4, 64, 255, -1, 1, False), (8, 4, 64, 256, -1, 1, True),
                                                              (4, 2, 128, 300, 239, 1, False), (4, 2, 128, 300, 240, 1, True), (16, 8, 64, 320, -1, 1, False), (16, 8, 64, 384, -1, 1, True),
                                                              (16, 8, 64, 256, -1, 1, True), (3, 3, 64, 300, -1, 1, False)])
def test_where_prompt_attention_keeps_its_scores(heads, kv, d, seq, window, batch, kept):
    names = kernels_of(*models.build_gqa(batch, heads, kv, d, 0, seq, ir.F16, window, True, seed=1))
    assert ("gqa_prefill_scores" in names) == kept and ("gqa_prefill_tc" in names) != kept


@pytest.mark.parametrize("n", [40, 64, 200, 700])
def test_experts_with_more_small_tiles_than_ctas(n):
    """Tiles of 32 rows in four CTAs per SM, a CTA per tile and none for the tiles that the counts do not give; persistent ones where groups have many rows."""
    m = Experts("bf16", 264, 24, 3, 1100)
    m.check(m.rows(n))


@pytest.mark.parametrize("dtype,d,past,seq,alone", [(ir.F16, 32, 1, 1, False), (ir.F32, 256, 40, 3, False), (ir.F16, 64, 255, 1, False), (ir.F16, 64, 256, 1, True),
                                                    (ir.F32, 64, 251, 12, True), (ir.F16, 128, 100, 20, False)])
def test_small_caches_are_copied_beside_the_new_rows(dtype, d, past, seq, alone):
    """Up to 2^16 elements the launch that writes the new rows copies the past: bit for bit, zeros behind ragged rows, the line itself."""
    module, feed = models.build_gqa(2, 4, 2, d, past, seq, dtype, -1, True, seed=d + seq)
    valid = [past, past // 3]
    feed["seqlens_k"] = HostTensor.from_numpy(np.array([v + seq - 1 for v in valid], np.int32))
    assert ("gqa_copy_past" in kernels_of(module.clone(), feed)) == alone
    tol = dict(atol=4e-3, rtol=4e-3) if dtype == ir.F16 else dict(atol=2e-4, rtol=1e-3)
    got = {n: t.numpy() for n, t in differential(module, feed, **tol)[0]}
    for name in ("key", "value"):
        for b, v in enumerate(valid):
            assert np.array_equal(got["present_" + name][b, :, :v], feed["past_" + name].numpy()[b, :, :v])
            assert not got["present_" + name][b, :, v + seq:].any()


@pytest.mark.parametrize("model,vocab", [("c1", 300), ("1b", 130), ("1b", 131072), ("1b", 131073), ("1b", 300001)])
def test_logits_as_f32(model, vocab):
    """Logits of one chunk, of whole chunks and of a tail, widened as they land: the stored values themselves. The first step does not know how many there are."""
    cfg = models.config_c1() if model == "c1" else models.config_gemma3_1b()
    cfg.layers, cfg.vocab = 1, vocab
    module, ids = models.build_decoder(cfg, seed=3), [5, 7, 11]
    a, b = (llm.NativeLlmSession(cuda_backend(), module.clone(), 16) for _ in range(2))
    for i in ids:
        raw, written = np.empty(4 * vocab, np.uint8), ctypes.c_size_t()
        assert a._lib.ox_llm_step(a._h, (ctypes.c_int64 * 1)(i), 1, None, raw.ctypes.data_as(ctypes.c_void_p), raw.size, ctypes.byref(written)) == 0
        want = raw[:written.value].view(np.float32 if model == "c1" else np.float16).astype(np.float32)
        got = b.step_logits([i])
        assert got.shape == (vocab,) and np.array_equal(got, want)


@pytest.mark.parametrize("heads,kv,dim,vdim,window,softcap,rising", [(4, 1, 256, 256, 0, 30.0, 0.0), (20, 1, 72, 136, 100, 0.0, 0.0), (3, 3, 128, 64, 0, 0.0, 0.3), (2, 1, 192, 200, 65, 0.0, 0.3),
                                                                    (64, 1, 64, 64, 0, 4.0, 0.0), (5, 5, 16, 8, 1, 0.0, 0.0)])
def test_prompts_over_pages_in_tensor_memory(heads, kv, dim, vdim, window, softcap, rising):
    """Unwritten places of the pools hold no numbers. Tiles of 128 rows that heads do not fill evenly, two tokens per tile, portions that begin inside a page, windows that leave
    tiles out, sums in either place of the tensor memory; scores that rise by more than 2^8 within a row, so that the sums are taken against a new maximum."""
    T = 330
    a = Attention("bf16", heads, kv, dim, vdim, scale=1.0 if rising else 2.0 / np.sqrt(dim), softcap=softcap, window=window, norm=int(not rising), sink=int(not rising))
    a.pools = [a.s.upload(act(np.full((40, kv, 64, d), np.nan), ir.BF16)) for d in (dim, vdim)]
    q, k, v = a.random(T)
    if rising:
        k = to_bf16(0.05 * k)
        q[..., 0], k[..., 0] = 1.0, to_bf16(rising * np.arange(T))[:, None]
    x, want, got, at = (q, k, v), a.want(q, k, v), [], 0
    a.s.enable_profiling(True)
    for n in (2, 129, 70, T - 201):
        got.append(a.step([(0, *piece(x, at, at + n)), (8, *piece(x, at, at + 5))])[0])
        at += n
    assert any("paged_kv_prefill" == kernel for kernel, _, _ in a.s.take_timings())
    err = row_err(np.concatenate(got), want)
    assert np.isfinite(err).all() and err.max() < 1.5e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("heads,kv,dim,far", [(32, 16, 128, 128), (20, 1, 72, 40), (2, 1, 256, 300)])
def test_prompts_whose_keys_are_their_values(heads, kv, dim, far):
    """Unwritten places of the pool and of its factors hold no numbers; tiles nearer than the farthest addend, across it and behind it; three tiles in the ring."""
    r, T, rows = np.random.default_rng(dim), 420, 12
    q, k = to_bf16(r.standard_normal((T, heads, dim))), to_bf16(r.standard_normal((T, kv, dim)))
    q_w, k_w, bias = to_bf16(1 + 0.3 * r.standard_normal(heads * dim)), to_bf16(1 + 0.3 * r.standard_normal(kv * dim)), r.standard_normal((rows, heads))
    kw = dict(scale=2.0 / np.sqrt(dim), temp=(0.4, 30))
    a = test_gpu_lovuzen.Attention("bf16", heads, kv, dim, lovuzen.distance_bias(bias, far), q_w, k_w, **kw)
    a.pool = a.s.upload(act(np.full(a.pool.shape, np.nan), ir.BF16))
    a.scales = a.s.upload(HostTensor.from_numpy(np.full(a.scales.shape, np.nan, np.float32)))
    got, at = [], 0
    for n in (3, 130, T - 133):
        got.append(a.step([(0, q[at:at + n], k[at:at + n]), (8, q[at:at + 5], k[at:at + 5])])[0])
        at += n
    got, want = np.concatenate(got), attention_want(q, k, bias, far, q_w, k_w, **kw)
    err = np.sqrt(((got - want) ** 2).mean(axis=(1, 2))) / np.sqrt((want ** 2).mean())
    assert np.isfinite(err).all() and err.max() < 1e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("form,heads,dim,vdim", [("plain", 4, 64, 128), ("plain", 4, 128, 256), ("capped", 4, 128, 128), ("capped", 4, 64, 192), ("keys", 64, 64, 64), ("keys", 64, 128, 128), ("keys", 64, 192, 192)])
def test_prompts_whose_maxima_rise_for_some_rows(form, heads, dim, vdim):
    """Warps of one CTA that take a new maximum in every tile, and are late for it, beside warps that never do: one to four tiles, either place of the weights. The sums of
    the others have to wait for the tile before the last as well. Every run gives the same bits."""
    r, T = np.random.default_rng(dim + vdim), 256
    place, tile = np.arange(T), np.arange(T) // 64
    k, v = to_bf16(0.1 * r.standard_normal((T, 1, dim))), to_bf16(r.standard_normal((T, 1, vdim)))
    q = to_bf16(0.1 * r.standard_normal((T, heads, dim)))
    if form == "keys":  # 64 heads: a warp's rows are half of a token's; their addends fall with the distance
        bias = np.zeros((heads, T), np.float32)
        bias[:32] = -0.25 * np.arange(T)
        a = test_gpu_lovuzen.Attention("bf16", heads, 1, dim, bias, np.ones(heads * dim, np.float32), np.ones(dim, np.float32), scale=0.2)
        qn, kn = (ref.rms_norm(x.reshape(T, -1).astype(np.float64), 1.0, 1e-5).reshape(x.shape) for x in (q, k))
        far = np.maximum(place[:, None] - place[None], 0)
        score, v, x = np.einsum("thd,jd->htj", qn, kn[:, 0]) * 0.2 + bias[:, far], k, (q, k)
    else:  # four heads: a warp's rows are eight tokens'; every other eight see scores that rise by 10 from tile to tile
        a = Attention("bf16", heads, 1, dim, vdim, scale=1.0, softcap=60.0 if form == "capped" else 0.0, norm=0, sink=0)
        q[..., 0], k[..., 0] = (place // 8 % 2)[:, None], (10 * tile)[:, None]
        score, x = np.einsum("thd,jd->htj", q.astype(np.float64), k[:, 0].astype(np.float64)), (q, k, v)
        if form == "capped":
            score = 60.0 * np.tanh(score / 60.0)
    score = np.where(place[None] <= place[:, None], score, -np.inf)
    w = np.exp(score - score.max(-1, keepdims=True))
    want = np.einsum("htj,jd->thd", w / w.sum(-1, keepdims=True), v[:, 0].astype(np.float64))
    first = None
    for run in range(60):
        got = a.step([(0, *x)])[0]
        first = got if first is None else first
        assert np.array_equal(got, first), run
        a.past.pop(0)  # the same pages once more
    err = row_err(first, want)
    assert err.max() < 1.5e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("width", [4, 1020, 1028, 3072, 4100, 6144, 6148])
def test_residual_norms_of_rows_in_registers(width):
    """Widths at the ends of a thread's packs and beyond them; everything that a norm in front of or behind the sum can take. f32 sums of at most 6148 squares."""
    r, rows, of, eps = np.random.default_rng(width), 5, HostTensor.from_numpy, 1e-4
    t = {n: r.standard_normal((rows, width)).astype(np.float32) for n in ("y", "res", "add", "gate")}
    v = {n: (1 + 0.2 * r.standard_normal(width)).astype(np.float32) for n in ("w", "gain", "post", "offset")}
    x = {n: a.astype(np.float64) for n, a in {**t, **v}.items()}
    for pre in (0, 1):
        b = ir.GraphBuilder()
        i = {n: b.input(n, ir.F32, [rows, width]) for n in t}
        if pre:
            ins, attrs = [i["y"], b.constant(of(v["w"])), i["res"], b.constant(of(v["post"])), i["add"], b.constant(of(v["offset"]))], {"residual": 1, "post": 1, "add": 1, "offset": 1, "add_scale": 0.3}
            want = ref.rms_norm(ref.rms_norm(x["y"], x["post"], eps) + x["res"] + 0.3 * x["add"] + x["offset"], x["w"], eps)
        else:
            ins, attrs = [i["y"], b.constant(of(v["w"])), i["res"], b.constant(of(v["gain"])), i["gate"]], {"residual": 1, "gain": 1, "gate": 1, "gate_offset": 0}
            want = ref.rms_norm(x["y"], x["w"], eps) * x["gain"] * x["gate"] + x["res"]
        b.output("out", b.composite("onyxia.ResidualNorm", dict(attrs, epsilon=eps, pre=pre), ins, [(ir.F32, [rows, width])])[0])
        got = be.run_once(cuda_backend(), b.finish(), {n: of(a) for n, a in t.items()})[0][1].numpy()
        assert rel_err(got, want) < 1e-6, pre


@pytest.mark.parametrize("dtype,shape,axis", [(np.float16, (50, 24), 0), (np.float16, (50, 23), 0), (np.int64, (7, 2), 0), (np.int64, (7, 3), 0), (np.uint8, (9, 16), 0), (np.uint8, (9, 5), 0),
                                              (np.float32, (3, 11, 8), 1), (np.float32, (3, 11, 6), 1), (np.float32, (6, 40), 1), (np.float16, (5, 7000), 0)])
def test_slices_gathered_in_units(dtype, shape, axis):
    """Slices of whole 16-byte units and others, along the first axis and behind it, indexes counted from the end."""
    r = np.random.default_rng(len(shape))
    data, idx = r.integers(0, 100, shape).astype(dtype), r.integers(-shape[axis], shape[axis], (3, 7)).astype(np.int64)
    b = ir.GraphBuilder()
    b.output("y", b.gather(b.constant(HostTensor.from_numpy(data)), b.input("i", ir.I64, [3, 7]), axis=axis))
    got = be.run_once(cuda_backend(), b.finish(), {"i": HostTensor.from_numpy(idx)})[0][1].numpy()
    assert np.array_equal(got, np.take(data, np.where(idx < 0, idx + shape[axis], idx), axis=axis))


@pytest.mark.parametrize("width", [8, 264, 2056, 8192, 8200, 12])
def test_norms_of_eights(width):
    """Rows of one group of eight, of a part of a warp, of all threads, and those that other kernels take: the oracle's bits, also of squares that overflow and of what is no number."""
    r = np.random.default_rng(width)
    x, w = (4 * r.standard_normal((6, width))).astype(np.float16), (1 + 0.1 * r.standard_normal(width)).astype(np.float16)
    x[1, width // 2], x[2, 0], x[3, width - 1], x[4] = 300.0, np.inf, np.nan, 0.0
    b = ir.GraphBuilder()
    b.output("y", b.composite("SimplifiedLayerNormalization", {"epsilon": 1e-6}, [b.input("x", ir.F16, list(x.shape)), b.input("w", ir.F16, [width])], [(ir.F16, list(x.shape))])[0])
    module, feed = b.finish(), {"x": HostTensor.from_numpy(x), "w": HostTensor.from_numpy(w)}
    got, want = be.run_once(cuda_backend(), module.clone(), feed)[0][1].numpy(), be.run_once(oracle.RefBackend(), module, feed)[0][1].numpy()
    assert np.array_equal(got, want, equal_nan=True)


def prompt_over_pages(op, attrs, rows, before, pools, after, out, portions):
    """A prompt in portions through one attention node in bf16 whose pools hold no numbers yet: its results and the kernels that ran. `before` and `after`: constants around the
    pools and the description of the step; `out`: heads and their width."""
    b = ir.GraphBuilder()
    N, R, TW, n_pages = b.sym("n"), b.sym("r"), b.sym("w"), pools[0][1][0]
    ins = [b.input("proj", ir.BF16, [N, rows.shape[1]])] + [b.constant(HostTensor.from_numpy(np.asarray(c, np.float32))) for c in before]
    ins += [b.input(f"pool{i}", dt, shape) for i, (dt, shape) in enumerate(pools)] + [b.input("seqs", ir.I32, [R, 4]), b.input("table", ir.I32, [R, TW])]
    outs = b.composite(op, attrs, ins + [b.constant(HostTensor.from_numpy(np.asarray(c, np.float32))) for c in after], [(ir.BF16, [N, out[0] * out[1]])] + pools)
    for i, v in enumerate(outs):
        b.output(f"out{i}", v)
    s = cuda_backend().prepare(b.finish())
    held = [s.upload(act(np.full(shape, np.nan), dt)) for dt, shape in pools]
    table = s.upload(HostTensor.from_numpy(np.random.default_rng(0).permutation(n_pages).astype(np.int32)[None]))
    s.enable_profiling(True)
    got, at = [], 0
    for n in portions:
        feed = {"proj": s.upload(act(rows[at:at + n], ir.BF16)), "seqs": s.upload(HostTensor.from_numpy(np.array([[0, n, at, 0]], np.int32))), "table": table}
        o = dict(s.run({**feed, **{f"pool{i}": t for i, t in enumerate(held)}}))
        got.append(s.download(o["out0"]).numpy())
        held, at = [o[f"out{i + 1}"] for i in range(len(pools))], at + n
    return np.concatenate(got).reshape(-1, *out), {kernel for kernel, _, _ in s.take_timings()}


@pytest.mark.parametrize("page", [16, 32, 64])
@pytest.mark.parametrize("heads,kv,dim,vdim,window,softcap", [(4, 2, 72, 136, 50, 0.0), (16, 1, 256, 256, 0, 30.0), (3, 3, 16, 8, 0, 0.0)])
def test_prompts_over_pages_of_any_size(page, heads, kv, dim, vdim, window, softcap):
    """Tiles of 64 keys over several pages take the `mma.sync` kernel."""
    r, T, scale = np.random.default_rng(page), 200, 2.0 / np.sqrt(dim)
    q, k, v = (to_bf16(r.standard_normal((T, n, d))) for n, d in ((heads, dim), (kv, dim), (kv, vdim)))
    attrs = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "rot_dims": 0, "window": window, "scale": scale, "softcap": softcap, "epsilon": 1e-5, "norm": 0, "sink": 1,
             "q_offset": 0, "k_offset": heads * dim, "v_offset": (heads + kv) * dim}
    rows = np.concatenate([x.reshape(T, -1) for x in (q, k, v)], axis=1)
    n = 256 // page
    got, kernels = prompt_over_pages("onyxia.PagedKVAttention", attrs, rows, [kipizen.turns_per_position(0, 100.0, 1.0)], [(ir.BF16, [n, kv, page, d]) for d in (dim, vdim)], [],
                                     (heads, vdim), (3, 130, 67))
    assert ("paged_kv_prefill" in kernels) == (page == 64) and ("paged_kv_prefill_mma" in kernels) == (page < 64)
    err = row_err(got, kipizen_ref.attention(*(x.astype(np.float64) for x in (q, k, v)), scale, softcap or None, window or None))
    assert np.isfinite(err).all() and err.max() < 1.5e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("page,heads,kv,dim,far", [(16, 32, 16, 128, 128), (32, 20, 1, 72, 40), (16, 2, 1, 256, 300), (64, 20, 1, 72, 40), (64, 8, 1, 64, 5500)])
def test_prompts_whose_keys_are_their_values_over_pages_of_any_size(page, heads, kv, dim, far):
    """Pages of less than 64 keys, and more addends by distance than stand beside the tiles in shared memory, take the `mma.sync` kernel."""
    r, T, kw = np.random.default_rng(page), 200, dict(scale=2.0 / np.sqrt(dim), temp=(0.4, 30))
    q, k = (to_bf16(r.standard_normal((T, n, dim))) for n in (heads, kv))
    q_w, k_w, bias = to_bf16(1 + 0.3 * r.standard_normal(heads * dim)), to_bf16(1 + 0.3 * r.standard_normal(kv * dim)), r.standard_normal((12, heads))
    attrs = {"heads": heads, "kv_heads": kv, "dim": dim, "q_offset": 0, "k_offset": heads * dim, "scale": kw["scale"], "epsilon": 1e-5, "temp_coef": 0.4, "temp_every": 30.0, "out_scale": 1.0}
    rows = np.concatenate([x.reshape(T, -1) for x in (q, k)], axis=1)
    got, kernels = prompt_over_pages("onyxia.PagedAttention", attrs, rows, [q_w, k_w, lovuzen.distance_bias(bias, far)], [(ir.BF16, [256 // page, kv, page, dim]), (ir.F32, [256 // page, page])],
                                     [], (heads, dim), (3, 130, 67))
    mma = page < 64 or far == 5500
    assert ("paged_attn_prefill_mma" in kernels) == mma and ("paged_attn_prefill" in kernels) == (not mma)
    want = attention_want(q, k, bias, far, q_w, k_w, **kw)
    err = np.sqrt(((got - want) ** 2).mean(axis=(1, 2))) / np.sqrt((want ** 2).mean())
    assert np.isfinite(err).all() and err.max() < 1e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("page", [16, 32, 64])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(4, 2, 64, 128), (20, 1, 72, 136)])
def test_mixed_heads_over_pages_of_any_size(page, heads, kv, dim, vdim):
    """The softmax's sums alone come from the `mma.sync` kernel where a tile lies in several pages."""
    r, T, scale = np.random.default_rng(page), 200, 1.5 / np.sqrt(dim)
    q, k, v = (to_bf16(r.standard_normal((T, n, d))) for n, d in ((heads, dim), (kv, dim), (kv, vdim)))
    temp, talk = to_bf16(r.uniform(0.5, 2, heads)), to_bf16(0.6 * np.eye(heads) + 0.5 * r.standard_normal((heads, heads)) / np.sqrt(heads))
    attrs = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "rot_dims": 0, "scale": scale, "temps": 1, "talk": 1, "q_offset": 0, "k_offset": heads * dim, "v_offset": (heads + kv) * dim}
    rows = np.concatenate([x.reshape(T, -1) for x in (q, k, v)], axis=1)
    got, kernels = prompt_over_pages("onyxia.PagedKVAttention", attrs, rows, [kipizen.turns_per_position(0, 100.0, 1.0)], [(ir.BF16, [256 // page, kv, page, d]) for d in (dim, vdim)],
                                     [temp, talk], (heads, vdim), (3, 130, 67))
    assert ("talk_lse" in kernels) == (page == 64) and ("talk_lse_mma" in kernels) == (page < 64)
    err = row_err(got, ref.talking_attention(*(x.astype(np.float64) for x in (q, k, v)), scale, temp.astype(np.float64), talk.astype(np.float64)))
    assert np.isfinite(err).all() and err.max() < 2e-2, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("more", [0, 1, 2400])
@pytest.mark.parametrize("scores", ["chosen", "corrected"])
def test_routing_in_one_round_and_more(more, scores):
    """A warp per token as long as every SM has one CTA at most, two tokens per warp beyond; the last CTA has one token."""
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count + more
    m = Experts("bf16", 64, 8, 2, 40) if scores == "chosen" else test_gpu_mufevik.Experts("bf16", 64, 8, 2, 40, (4, 2), 72, correction=0.2 / 8)
    m.s.enable_profiling(True)
    m.check(m.rows(n))
    kernels = {kernel for kernel, _, _ in m.s.take_timings()}
    assert ("moe_route" in kernels) == (more == 0) and ("moe_route_pairs" in kernels) == (more > 0)


@pytest.mark.parametrize("form,vdim", [("plain", 128), ("plain", 256), ("capped", 64), ("sink", 128), ("keys", 64)])
def test_prompts_where_one_late_key_stands_out(form, vdim):
    """A key of the second tile that weighs 2^7.4 of the first tile's only key, between two bf16 values. Taken against the maximum it weighs 1, and only the other key's share of
    2^-7.4 is rounded, by 2^-8 of it and less: results differ from the rounded exact ones where these are that close to the middle of two bf16 values, 1 % of them. (Taken against
    the first tile's maximum: off by 2.8e-3 of a value, with 3.9e-3 … 7.8e-3 between two values, so four in ten.)"""
    r, T, heads, dim, late = np.random.default_rng(vdim), 128, 4, 64, 5.15625
    v, place = to_bf16(r.standard_normal((T, 1, vdim))), np.arange(T)
    if form == "keys":
        bias = np.full((heads, T), -100.0, np.float32)
        bias[:, 0], bias[:, 64] = late, 0.0
        a = test_gpu_lovuzen.Attention("bf16", heads, 1, dim, bias, np.ones(heads * dim, np.float32), np.ones(dim, np.float32), scale=0.0)
        score = np.repeat(bias[0][np.maximum(place[:, None] - place[None], 0)][None], heads, axis=0)
        x = (to_bf16(r.standard_normal((T, heads, dim))), v)
    else:
        cap, shift = 600.0 if form == "capped" else 0.0, 5.0 if form == "sink" else 0.0
        a = Attention("bf16", heads, 1, dim, vdim, scale=1.0, softcap=cap, norm=0, sink=int(form == "sink"))
        q, k = np.zeros((T, heads, dim), np.float32), np.zeros((T, 1, dim), np.float32)
        q[..., 0], k[:, 0, 0] = 1.0, -100.0
        k[0, 0, 0], k[64, 0, 0] = -shift, late - shift
        score, x = np.einsum("thd,jd->htj", q.astype(np.float64), k[:, 0].astype(np.float64)), (q, k, v)
        if cap:
            score = cap * np.tanh(score / cap)
    w = np.where(place[None] <= place[:, None], np.exp(score), 0.0)
    want = np.einsum("htj,jd->thd", w / (w.sum(-1, keepdims=True) + (form == "sink")), v[:, 0].astype(np.float64))[64:]
    got = a.step([(0, *x)])[0][64:]
    assert (got != to_bf16(want)).mean() < 0.05


@pytest.mark.parametrize("rows,k,n", [(303, 2560, 2560), (200, 2560, 4160), (2048, 6912, 1152)])
def test_results_of_cut_chains(rows, k, n):
    """A chain of tensor-core sums is 6.7e-8 off per 64 k; cut into two pieces and more, half of that and less."""
    r = np.random.default_rng(rows)
    x, w = to_bf16(r.standard_normal((rows, k), dtype=np.float32)), to_bf16(r.standard_normal((n, k), dtype=np.float32) / np.sqrt(k))
    want = x.astype(np.float64) @ w.T.astype(np.float64)
    assert rel_err(run_linear(ir.BF16, x, w).astype(np.float64), want) < 0.6 * 6.7e-8 * k / 64
    assert rel_err(run_linear(ir.BF16, x, w, out_dtype=ir.BF16).astype(np.float64), want) < 2.0 ** -9


@pytest.mark.parametrize("rows,k,n", [(1046, 5376, 514), (300, 21504, 270)])
def test_pairs_of_ctas_sum_as_single_ones_do(rows, k, n, monkeypatch):
    """Long chains as f32 results: the bits of linear_tc whose k is not cut, whatever the tile."""
    r, got = np.random.default_rng(rows), []
    x, w = to_bf16(r.standard_normal((rows, k), dtype=np.float32)), to_bf16(r.standard_normal((n, k), dtype=np.float32) / np.sqrt(k))
    for tile in ("128,1", "256,0", "240,0", "96,0"):
        monkeypatch.setenv("ONYXIA_LINEAR_TILE", tile)
        got.append(run_linear(ir.BF16, x, w))
    assert all(np.array_equal(got[0], g) for g in got[1:])
    assert rel_err(got[0].astype(np.float64), x.astype(np.float64) @ w.T.astype(np.float64)) < 2 * 6.7e-8 * k / 64


@pytest.mark.parametrize("kind", ["f32", "bf16"])
@pytest.mark.parametrize("dim,vdim", [(127, 10), (128, 128), (129, 7), (20, 129), (6, 130)])
def test_any_shape_by_one_or_two_threads_per_key(kind, dim, vdim):
    """Either side of a thread per value dimension, halves of a key that are no multiple of four, more than one chunk of 128 keys, prompts and single tokens."""
    a = Attention(kind, 3, 1, dim, vdim, scale=1.0 / np.sqrt(dim), norm=0, sink=1)
    x, got, at = a.random(200), [], 0
    want = a.want(*x)
    for n in (1, 126, 1, 1, 1, 70):
        got.append(a.step([(0, *piece(x, at, at + n))])[0])
        at += n
    err = row_err(np.concatenate(got), want)
    assert err.max() < (1e-5 if kind == "f32" else 1e-2), (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("form,heads,kv,tokens,mma", [("values", 4, 1, 64, True), ("values", 4, 1, 65, False), ("values", 3, 3, 65, False), ("keys", 4, 1, 64, True), ("keys", 4, 1, 65, False),
                                                      ("keys", 3, 3, 128, True), ("keys", 3, 3, 129, False), ("sums", 4, 2, 64, True), ("sums", 4, 2, 65, False)])
def test_where_prompts_are_short(form, heads, kv, tokens, mma):
    """Sequences of one page take the `mma.sync` kernel; heads that share no keys which are their values, of two."""
    r, dim, scale, page = np.random.default_rng(tokens), 64, 0.25, 64
    n = -(-tokens // page)
    q, k, v = (to_bf16(r.standard_normal((tokens, g, dim))) for g in (heads, kv, kv))
    turns, f64 = kipizen.turns_per_position(0, 100.0, 1.0), np.float64
    attrs = {"heads": heads, "kv_heads": kv, "dim": dim, "scale": scale, "q_offset": 0, "k_offset": heads * dim, "epsilon": 1e-5}
    values, pool = {"vdim": dim, "rot_dims": 0, "v_offset": (heads + kv) * dim}, (ir.BF16, [n, kv, page, dim])
    rows = np.concatenate([x.reshape(tokens, -1) for x in ((q, k) if form == "keys" else (q, k, v))], axis=1)
    if form == "keys":
        one, bias = np.ones(heads * dim, np.float32), r.standard_normal((12, heads))
        got, kernels = prompt_over_pages("onyxia.PagedAttention", dict(attrs, temp_coef=0.0, temp_every=0.0, out_scale=1.0), rows, [one, one[:kv * dim], lovuzen.distance_bias(bias, 40)],
                                         [pool, (ir.F32, [n, page])], [], (heads, dim), (tokens,))
        want, name = attention_want(q, k, bias, 40, one, one[:kv * dim], scale=scale), "paged_attn_prefill"
    elif form == "values":
        got, kernels = prompt_over_pages("onyxia.PagedKVAttention", dict(attrs, **values, window=0, softcap=0.0, norm=0, sink=0), rows, [turns], [pool, pool], [], (heads, dim), (tokens,))
        want, name = kipizen_ref.attention(q.astype(f64), k.astype(f64), v.astype(f64), scale, sink=False), "paged_kv_prefill"
    else:
        temp, talk = to_bf16(r.uniform(0.5, 2, heads)), to_bf16(np.eye(heads) + 0.3 * r.standard_normal((heads, heads)))
        got, kernels = prompt_over_pages("onyxia.PagedKVAttention", dict(attrs, **values, temps=1, talk=1), rows, [turns], [pool, pool], [temp, talk], (heads, dim), (tokens,))
        want, name = ref.talking_attention(q.astype(f64), k.astype(f64), v.astype(f64), scale, temp.astype(f64), talk.astype(f64)), "talk_lse"
    assert (name + "_mma" in kernels) == mma and (name in kernels) == (not mma)
    err = row_err(got, want)
    assert np.isfinite(err).all() and err.max() < 2e-2, (int(err.argmax()), float(err.max()))
