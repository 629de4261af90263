"""GPU parity of the device-resident cache and the fused decode attention,
through the C ABI, against the oracle and the reference-made golden vectors.

Tolerances: fp32 activations 1e-5; bf16 activations 2e-3, on the error of a
(unit, head) output row relative to the row's largest reference element,
max|out-ref| / max|ref| (`rel_err`).  The tests also print the element-wise
figure max |out-ref| / max(|ref|, 1e-3 * max|ref| of the row) (`elem_err`),
which weighs the same absolute error against each element's own magnitude."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import kivi_oracle as ko

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-5
TOL_BF16 = 2e-3


@pytest.fixture(scope="module")
def cabi():
    from intel_kivi_hybrid_b200 import cabi as m
    return m


def rel_err(out, ref):
    out, ref = out.float().cpu(), ref.float().cpu()
    num = (out - ref).abs().amax(dim=-1)
    den = ref.abs().amax(dim=-1).clamp_min(1e-30)
    return float((num / den).max())


def elem_err(out, ref):
    out, ref = out.float().cpu(), ref.float().cpu()
    floor = 1e-3 * ref.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)
    return float(((out - ref).abs() / torch.maximum(ref.abs(), floor)).max())


def units(x):            # [B,H,T,D] -> [B*H,T,D]
    return x.reshape(x.shape[0] * x.shape[1], *x.shape[2:])


def test_state_machine_matches_reference_cache(cabi, golden_dir):
    sm = np.load(os.path.join(golden_dir, "state_machine_vectors.npz"))
    K, V = torch.from_numpy(sm["long__K"]), torch.from_numpy(sm["long__V"])
    st = cabi.LayerStore(3, 64, 32, 128, 512, torch.float32, "cuda")
    Kc, Vc = units(K).cuda(), units(V).cuda()
    st.update(Kc[:, :200], Vc[:, :200], cabi.ROUND_HALF_EVEN)
    assert (st.quant_len, st.res_len) == (96, 104)
    for t in range(200, 300):
        st.update(Kc[:, t:t + 1], Vc[:, t:t + 1], cabi.ROUND_HALF_EVEN)
    assert st.quant_len == int(sm["long__quant_tokens"])
    k, v = st.materialize()
    assert torch.equal(k.cpu().reshape(1, 3, -1, 64), torch.from_numpy(sm["long__served_k"]))
    assert torch.equal(v.cpu().reshape(1, 3, -1, 64), torch.from_numpy(sm["long__served_v"]))


def test_small_g_state_machine_matches_reference_cache(cabi, golden_dir):
    sm = np.load(os.path.join(golden_dir, "state_machine_vectors.npz"))
    steps, prefill, G, R, D, layers, heads = [int(v) for v in sm["params"]]
    for i in range(layers):
        truth = torch.from_numpy(sm[f"in_place__truth_k{i}"])
        tk = units(truth).cuda()
        tv = (2 * torch.arange(truth.shape[2]).view(1, 1, -1, 1).float() - truth)
        tv = units(tv).cuda()
        st = cabi.LayerStore(heads, D, G, R, 64, torch.float32, "cuda")
        st.update(tk[:, :prefill], tv[:, :prefill], cabi.ROUND_HALF_EVEN)
        for t in range(prefill, prefill + steps):
            st.update(tk[:, t:t + 1], tv[:, t:t + 1], cabi.ROUND_HALF_EVEN)
        k, _ = st.materialize()
        assert torch.equal(k.cpu().reshape(1, heads, -1, D), torch.from_numpy(sm[f"in_place__served_k{i}"]))
        assert st.quant_len == int(sm["in_place__quant_tokens"][i])


def test_packed_store_matches_oracle_flush_by_flush(cabi):
    B, H, D, G, R = 1, 4, 64, 32, 128
    K = ko.make_keys(B, H, 300, D, seed=21)
    V = ko.make_values(B, H, 300, D, seed=21)
    oc = ko.OracleCache(D, G, R, rounding="half_away")
    st = cabi.LayerStore(B * H, D, G, R, 512, torch.float32, "cuda")
    Kc, Vc = units(K).cuda(), units(V).cuda()
    oc.append(K[:, :, :150], V[:, :, :150]); st.update(Kc[:, :150], Vc[:, :150])
    for t in range(150, 300):
        oc.append(K[:, :, t:t + 1], V[:, :, t:t + 1]); st.update(Kc[:, t:t + 1], Vc[:, t:t + 1])
    assert st.quant_len == oc.quantized_len and st.res_len == oc.residual_len
    ng = st.quant_len // G
    ks = torch.stack(oc.k_scales, dim=2).reshape(B * H, ng, D)
    kz = torch.stack(oc.k_zeros, dim=2).reshape(B * H, ng, D)
    assert torch.equal(st.k_scales[:, :ng].cpu(), ks) and torch.equal(st.k_zeros[:, :ng].cpu(), kz)
    vs = torch.cat(oc.v_scales, dim=2).reshape(B * H, ng * G, D // G)
    assert torch.equal(st.v_scales[:, :ng * G].cpu(), vs)
    vp = torch.cat(oc.v_packed, dim=2).reshape(B * H, ng * G, D // 4)
    assert torch.equal(st.v_codes[:, :ng * G].cpu(), vp)
    # key blocks hold the same codes as the reference layout, re-laid out
    kc = ko.unpack_codes(torch.stack(oc.k_packed, dim=2).reshape(B * H, ng, D, G // 4))   # [u,g,D,G]
    blk = st.k_codes[:, :ng].cpu().reshape(B * H, ng, G // 4, D)                            # one 64-wide half: [j][p(d)]
    perm = torch.tensor([(d & 3) | (((d >> 4) & 3) << 2) | (((d >> 2) & 3) << 4) for d in range(D)])
    blk = blk[..., perm]                                                                    # -> [j][d]
    Q = G // 4
    for e in range(4):
        got = (blk >> (2 * e)) & 3                       # bit pair e of byte j = token 4j + e
        assert torch.equal(got.transpose(2, 3), kc[..., e::4].to(torch.uint8))
    # served tensors: history round trip + exact residual
    k, v = st.materialize()
    sk, sv = oc.served()
    assert torch.equal(k.cpu(), units(sk)) and torch.equal(v.cpu(), units(sv))


def test_value_blocks_of_llama_shaped_layers_hold_the_reference_bytes(cabi):
    """D=128, G=32 layers store each 32-token value group as a re-laid block;
    undoing the documented permutation must give the reference's packed rows, and
    the served tensors must equal the oracle's bit for bit."""
    B, H, D, G, R = 1, 2, 128, 32, 128
    K = ko.make_keys(B, H, 200, D, seed=8)
    V = ko.make_values(B, H, 200, D, seed=8)
    oc = ko.OracleCache(D, G, R, rounding="half_away")
    st = cabi.LayerStore(B * H, D, G, R, 256, torch.float32, "cuda")
    oc.append(K, V); st.update(units(K).cuda(), units(V).cuda())
    ng = st.quant_len // G
    assert ng == oc.flushes == 3
    vp = torch.cat(oc.v_packed, dim=2).reshape(B * H, ng, G, D // 4)               # natural rows [t][b]
    blk = st.v_codes[:, :ng * G].cpu().reshape(B * H, ng, 4, 2, 8, 4, 4)            # [gd][kappa][r][c][n]
    nat = blk.permute(0, 1, 3, 5, 6, 2, 4).reshape(B * H, ng, G, D // 4)            # t = 16k+4c+n, b = 8gd+r
    assert torch.equal(nat, vp)
    vs = torch.cat(oc.v_scales, dim=2).reshape(B * H, ng, G, D // G)
    rows = st.v_scales[:, :ng * G].cpu().reshape(B * H, ng, 2, 4, 4, D // G)        # [kappa][n][c]
    assert torch.equal(rows.permute(0, 1, 2, 4, 3, 5).reshape(B * H, ng, G, D // G), vs)
    k, v = st.materialize()
    sk, sv = oc.served()
    assert torch.equal(k.cpu(), units(sk)) and torch.equal(v.cpu(), units(sv))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rounding", ["half_away", "half_even"])
def test_chunked_bulk_prefill_mixes_ring_and_new_tensor_groups(cabi, dtype, rounding):
    """Bulk updates whose first groups still hold ring tokens (virtual-sequence
    kernels) and whose remaining groups are cut straight out of the new tensor
    (direct kernels), in ragged chunks; one key channel and one value group carry
    a range so large that the scale has no reciprocal (plain-division branch)."""
    B, H, D, G, R = 1, 3, 128, 32, 128
    chunks = [50, 333, 1, 700, 95]
    T = sum(chunks)
    K = ko.make_keys(B, H, T, D, seed=5)
    V = ko.make_values(B, H, T, D, seed=6)
    K[0, 1, 400:420, 7] = 1.6e38; K[0, 1, 420:440, 7] = -1.6e38
    V[0, 2, 500, 32:48] = 1.6e38; V[0, 2, 500, 48:64] = -1.6e38
    if dtype == torch.bfloat16:
        K, V = K.bfloat16().float(), V.bfloat16().float()
    oc = ko.OracleCache(D, G, R, rounding=rounding)
    st = cabi.LayerStore(B * H, D, G, R, 1184, dtype, "cuda")
    mode = cabi.ROUND_HALF_EVEN if rounding == "half_even" else cabi.ROUND_HALF_AWAY
    Kc, Vc = units(K).cuda().to(dtype), units(V).cuda().to(dtype)
    t = 0
    for n in chunks:
        oc.append(K[:, :, t:t + n], V[:, :, t:t + n])
        st.update(Kc[:, t:t + n], Vc[:, t:t + n], mode)
        t += n
        assert st.quant_len == oc.quantized_len and st.res_len == oc.residual_len
    ng = st.quant_len // G
    ks = torch.stack(oc.k_scales, dim=2).reshape(B * H, ng, D)
    kz = torch.stack(oc.k_zeros, dim=2).reshape(B * H, ng, D)
    assert torch.equal(st.k_scales[:, :ng].cpu(), ks) and torch.equal(st.k_zeros[:, :ng].cpu(), kz)
    assert float(ks.max()) >= 1e30
    k, v = st.materialize()
    sk, sv = oc.served()
    assert torch.equal(k.cpu(), units(sk)) and torch.equal(v.cpu(), units(sv))


def test_import_keys_from_operator_layout(cabi):
    B, H, D, G, S = 1, 2, 128, 32, 96
    K = ko.make_keys(B, H, S, D, seed=3)
    kt = units(K).transpose(1, 2).contiguous().cuda()          # [u, D, S]
    packed = torch.empty(B * H, D, S // 4, dtype=torch.uint8, device="cuda")
    scales = torch.empty(B * H, D, S // G, device="cuda")
    zeros = torch.empty(B * H, D, S // G, device="cuda")
    cabi.quantize_keys(kt, packed, scales, zeros, G)
    a = cabi.LayerStore(B * H, D, G, 128, S, torch.float32, "cuda")
    a.import_keys(packed, scales, zeros, S)
    b = cabi.LayerStore(B * H, D, G, 128, S, torch.float32, "cuda")
    cabi.load_state(b, units(K).cuda(), units(K).cuda(), S)
    assert torch.equal(a.k_codes, b.k_codes) and torch.equal(a.k_scales, b.k_scales) and torch.equal(a.k_zeros, b.k_zeros)


def _attention_case(cabi, B, Hkv, n_rep, D, G, R, n_quant, n_res, dtype, seed, path, num_splits=0,
                    res_start=0, out_dtype=torch.float32):
    T = n_quant + n_res
    K = ko.make_keys(B, Hkv, T, D, seed).to(dtype)
    V = ko.make_values(B, Hkv, T, D, seed).to(dtype)
    q = ko.make_queries(B, Hkv * n_rep, D, seed).to(dtype)
    ref = ko.kivi_decode_attention(q, K, V, n_quant, G, "half_away")
    ref64 = ko.kivi_decode_attention(q, K, V, n_quant, G, "half_away", dtype=torch.float64)
    st = cabi.LayerStore(B * Hkv, D, G, R, max(n_quant, G), dtype, "cuda")
    cabi.load_state(st, units(K).cuda(), units(V).cuda(), n_quant)
    if res_start:                       # rotate the ring: same window, different slots
        st.k_res.copy_(torch.roll(st.k_res, res_start, dims=1))
        st.v_res.copy_(torch.roll(st.v_res, res_start, dims=1))
        st.res_start = res_start % R
    out = st.attention(q.cuda().contiguous(), n_rep=n_rep, num_splits=num_splits, path=path, out_dtype=out_dtype)
    torch.cuda.synchronize()
    assert torch.isfinite(out.float()).all()
    return rel_err(out, ref64.float()), rel_err(ref, ref64.float()), out, ref64


def test_attention_golden_seed42(cabi, golden_dir):
    av = np.load(os.path.join(golden_dir, "attention_vectors.npz"))
    q, k, v = (torch.from_numpy(av[n]) for n in ("query", "key", "value"))
    st = cabi.LayerStore(2, 64, 32, 128, 32, torch.float32, "cuda")
    cabi.load_state(st, units(k).cuda(), units(v).cuda(), 32, cabi.ROUND_HALF_EVEN)
    for i in range(q.shape[2]):
        out = st.attention(q[:, :, i].contiguous().cuda(), n_rep=1)
        assert rel_err(out, torch.from_numpy(av["out_kivi"])[:, :, i]) < TOL_F32


@pytest.mark.parametrize("n_quant,n_res,res_start", [(416, 96, 0), (608, 104, 40), (0, 77, 0), (96, 0, 0), (32, 1, 127)])
def test_attention_fp32_gpt2_shapes(cabi, n_quant, n_res, res_start):
    # config 0: B=1, H=12 (MHA), D=64, fp32, R=128, G=32
    err, oerr, _, _ = _attention_case(cabi, 1, 12, 1, 64, 32, 128, n_quant, n_res, torch.float32, 7,
                                      cabi.ATTN_FP32, res_start=res_start)
    print(f"[attn fp32 cfg0 q={n_quant} r={n_res}] rel err {err:.2e} (fp32 oracle vs fp64: {oerr:.2e})")
    assert err < TOL_F32


@pytest.mark.parametrize("D,G,n_rep", [(128, 32, 4), (128, 64, 2), (64, 16, 1), (128, 128, 8), (256, 32, 2), (32, 4, 3)])
def test_attention_fp32_shapes(cabi, D, G, n_rep):
    err, _, _, _ = _attention_case(cabi, 2, 2, n_rep, D, G, max(G, 64), 4 * G, max(G, 64) - 3, torch.float32, 11,
                                   cabi.ATTN_FP32)
    assert err < TOL_F32


@pytest.mark.parametrize("splits", [1, 2, 7, 31])
def test_attention_split_count_does_not_change_result(cabi, splits):
    err, _, out, _ = _attention_case(cabi, 1, 2, 4, 128, 32, 128, 31 * 32, 128, torch.float32, 5,
                                     cabi.ATTN_FP32, num_splits=splits)
    assert err < TOL_F32


@pytest.mark.parametrize("path,dtype,splits", [("fp32", torch.float32, 40), ("fp32", torch.float32, 100),
                                               ("mma", torch.bfloat16, 33), ("mma", torch.bfloat16, 70)])
def test_attention_with_more_than_32_partials_per_unit(cabi, path, dtype, splits):
    """The merge walks a row's partials 32 at a time, eight loads in flight: more
    than 32 pieces per unit (few units, long context) take its second round."""
    kernel = cabi.ATTN_FP32 if path == "fp32" else cabi.ATTN_MMA
    err, _, out, _ = _attention_case(cabi, 1, 2, 4, 128, 32, 128, 100 * 32, 128, dtype, 23, kernel, num_splits=splits)
    assert err < (TOL_F32 if dtype == torch.float32 else TOL_BF16)
    assert cabi.device_fault() == 0


def test_attention_bf16_llama_shape_fp32_kernel(cabi):
    # config 1 slice: GQA 4:1, D=128, bf16 activations, full ring
    err, _, _, _ = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_FP32)
    print(f"[attn bf16 cfg1 slice, fp32 kernel] rel err {err:.2e}")
    assert err < TOL_BF16
    err, _, _, _ = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_FP32,
                                   out_dtype=torch.bfloat16)
    assert err < 2 * TOL_BF16          # + half an ulp of the bf16 output itself


def test_attention_errors(cabi):
    st = cabi.LayerStore(2, 64, 32, 128, 64, torch.float32, "cuda")
    q = torch.randn(2, 1, 64, device="cuda")
    with pytest.raises(RuntimeError, match="empty"):
        st.attention(q)
    with pytest.raises(RuntimeError, match="no new tokens"):
        st.update(torch.empty(2, 0, 64, device="cuda"), torch.empty(2, 0, 64, device="cuda"))
    with pytest.raises(RuntimeError, match="overflow"):
        st.update(torch.randn(2, 400, 64, device="cuda"), torch.randn(2, 400, 64, device="cuda"))


# ---- tensor-core kernel ------------------------------------------------------

@pytest.mark.parametrize("n_quant,n_res,n_rep,splits", [
    (3968, 128, 4, 0), (32, 0, 4, 0), (64, 5, 4, 1), (96, 128, 4, 3), (2048 + 32, 100, 4, 5),
    (992, 128, 1, 0), (992, 128, 2, 2), (992, 128, 3, 0), (13 * 32, 96, 4, 13),
    (992, 128, 8, 0), (2048 + 32, 100, 5, 3), (96, 7, 6, 1), (64, 0, 7, 0)])
def test_attention_mma_bf16(cabi, n_quant, n_res, n_rep, splits):
    err, _, out, ref64 = _attention_case(cabi, 2, 4, n_rep, 128, 32, 128, n_quant, n_res, torch.bfloat16, 17,
                                         cabi.ATTN_MMA, num_splits=splits)
    print(f"[attn mma bf16 q={n_quant} r={n_res} rep={n_rep} splits={splits}] rel err {err:.2e}, "
          f"element-wise {elem_err(out, ref64.float()):.2e}")
    assert err < TOL_BF16
    assert cabi.device_fault() == 0


def test_attention_mma_matches_fp32_kernel_and_auto_dispatch(cabi):
    e_mma, _, o_mma, _ = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_MMA)
    e_auto, _, o_auto, _ = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_AUTO)
    e_f32, _, o_f32, _ = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_FP32)
    assert torch.equal(o_mma, o_auto)                 # bf16 queries dispatch to the tensor-core kernel
    _, _, _, ref64 = _attention_case(cabi, 2, 8, 4, 128, 32, 128, 3968, 128, torch.bfloat16, 13, cabi.ATTN_FP32)
    print(f"[attn cfg1 slice] mma {e_mma:.2e}  fp32 kernel {e_f32:.2e}  mma vs fp32 kernel {rel_err(o_mma, o_f32):.2e}; "
          f"element-wise: mma {elem_err(o_mma, ref64.float()):.2e}  fp32 kernel {elem_err(o_f32, ref64.float()):.2e}")
    assert e_mma < TOL_BF16 and rel_err(o_mma, o_f32) < TOL_BF16


def test_attention_mma_fp32_queries_and_bf16_output(cabi):
    err, _, _, _ = _attention_case(cabi, 1, 4, 4, 128, 32, 128, 1024, 64, torch.float32, 23, cabi.ATTN_MMA)
    print(f"[attn mma fp32 activations] rel err {err:.2e}")
    assert err < TOL_BF16
    err, _, _, _ = _attention_case(cabi, 1, 4, 4, 128, 32, 128, 1024, 64, torch.bfloat16, 23, cabi.ATTN_MMA,
                                   out_dtype=torch.bfloat16)
    assert err < 2 * TOL_BF16


def test_attention_mma_is_deterministic(cabi):
    _, _, a, _ = _attention_case(cabi, 2, 4, 4, 128, 32, 128, 2048, 128, torch.bfloat16, 3, cabi.ATTN_MMA)
    _, _, b, _ = _attention_case(cabi, 2, 4, 4, 128, 32, 128, 2048, 128, torch.bfloat16, 3, cabi.ATTN_MMA)
    assert torch.equal(a, b)


def test_attention_mma_rejects_other_shapes(cabi):
    st = cabi.LayerStore(2, 64, 32, 128, 64, torch.float32, "cuda")
    cabi.load_state(st, torch.randn(2, 64, 64, device="cuda"), torch.randn(2, 64, 64, device="cuda"), 64)
    with pytest.raises(RuntimeError, match="tensor-core path"):
        st.attention(torch.randn(2, 1, 64, device="cuda"), path=cabi.ATTN_MMA)


# ---- full-size properties (config 2 of the benchmark: 512 units x 32768 tokens) ----

def test_full_size_config2_properties(cabi):
    """At the benchmark's full size the oracle is too slow, so check properties that
    do not depend on size: the result does not depend on the number of splits, the
    tensor-core and the fp32 kernel agree, every output is a convex combination of
    value rows (inside their per-channel range), and a slice of units reproduces
    the CPU oracle."""
    B, Hkv, n_rep, D, G, R, n_quant, n_res = 64, 8, 4, 128, 32, 128, 32640, 128
    U, T = B * Hkv, n_quant + n_res
    g = torch.Generator(device="cuda").manual_seed(123)
    k = torch.empty(U, T, D, device="cuda", dtype=torch.bfloat16)
    v = torch.empty(U, T, D, device="cuda", dtype=torch.bfloat16)
    for u0 in range(0, U, 64):
        k[u0:u0 + 64] = torch.randn(64, T, D, device="cuda", generator=g).to(torch.bfloat16)
        v[u0:u0 + 64] = torch.randn(64, T, D, device="cuda", generator=g).to(torch.bfloat16)
    k[:, :, 5] *= 10.0                                     # an outlier channel
    st = cabi.LayerStore(U, D, G, R, n_quant, torch.bfloat16, "cuda")
    cabi.load_state(st, k, v, n_quant)
    q = torch.randn(U, n_rep, D, device="cuda", generator=g).to(torch.bfloat16)
    o_auto = st.attention(q, n_rep=n_rep, path=cabi.ATTN_MMA, out_dtype=torch.float32)
    o_s1 = st.attention(q, n_rep=n_rep, path=cabi.ATTN_MMA, num_splits=1, out_dtype=torch.float32)
    o_s9 = st.attention(q, n_rep=n_rep, path=cabi.ATTN_MMA, num_splits=9, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert cabi.device_fault() == 0 and torch.isfinite(o_auto).all()
    # different split counts change the running max that p = 2^(s-m) is taken against, hence the
    # fp16 rounding of p*s: agreement is at the level of that rounding, not bitwise
    e1, e9 = rel_err(o_s1, o_auto), rel_err(o_s9, o_auto)
    print(f"[cfg2 full size] splits 1 vs auto {e1:.2e}, 9 vs auto {e9:.2e}")
    assert e1 < TOL_BF16 and e9 < TOL_BF16
    # fp32 kernel on the last units (a full run of it takes ~5 ms; slicing needs a second store)
    sub = slice(U - 8, U)
    st8 = cabi.LayerStore(8, D, G, R, n_quant, torch.bfloat16, "cuda")
    cabi.load_state(st8, k[sub], v[sub], n_quant)
    o_f32 = st8.attention(q[sub].contiguous(), n_rep=n_rep, path=cabi.ATTN_FP32, out_dtype=torch.float32)
    print(f"[cfg2 full size] tensor-core vs fp32 kernel {rel_err(o_auto[sub], o_f32):.2e}")
    assert rel_err(o_auto[sub], o_f32) < TOL_BF16
    # convexity: the quantized values stay inside [min, max] of their group, so the output
    # stays inside the per-channel range of the unit's values
    vmin = v.float().amin(dim=1, keepdim=True)
    vmax = v.float().amax(dim=1, keepdim=True)
    eps = 1e-2
    assert bool(((o_auto >= vmin - eps) & (o_auto <= vmax + eps)).all())
    # oracle on the first KV head of the first batch row
    kk, vv = k[:1].cpu().reshape(1, 1, T, D), v[:1].cpu().reshape(1, 1, T, D)
    ref = ko.kivi_decode_attention(q[:1].cpu().reshape(1, n_rep, D), kk, vv, n_quant, G, "half_away", dtype=torch.float64)
    r0 = ref.float().reshape(1, n_rep, D)
    print(f"[cfg2 full size] unit 0 vs oracle: rel err {rel_err(o_auto[:1], r0):.2e}, element-wise {elem_err(o_auto[:1], r0):.2e}")
    assert rel_err(o_auto[:1], r0) < TOL_BF16


def test_full_size_config3_long_context(cabi):
    """The long-context shape: 32 units x (131072 quantized + 128 ring) tokens,
    bf16, split count chosen by the library (few units, so every unit is cut into
    many pieces).  One unit against the CPU oracle in fp64, agreement of the
    tensor-core and the fp32 kernel on two units, no bounded wait expired."""
    B, Hkv, n_rep, D, G, R, n_quant, n_res = 4, 8, 4, 128, 32, 128, 131072, 128
    U, T = B * Hkv, n_quant + n_res
    g = torch.Generator(device="cuda").manual_seed(321)
    k = torch.randn(U, T, D, device="cuda", generator=g)
    k[:, :, 17] *= 10.0
    k[:, :, 99] *= 10.0
    k = k.to(torch.bfloat16)
    v = torch.randn(U, T, D, device="cuda", generator=g)
    v *= 1.0 + 7.0 * (torch.rand(U, T, 1, device="cuda", generator=g) < 0.02)
    v = v.to(torch.bfloat16)
    st = cabi.LayerStore(U, D, G, R, n_quant, torch.bfloat16, "cuda")
    cabi.load_state(st, k, v, n_quant)
    q = torch.randn(U, n_rep, D, device="cuda", generator=g).to(torch.bfloat16)
    o_auto = st.attention(q, n_rep=n_rep, path=cabi.ATTN_MMA, out_dtype=torch.float32)
    o_s28 = st.attention(q, n_rep=n_rep, path=cabi.ATTN_MMA, num_splits=28, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert cabi.device_fault() == 0 and torch.isfinite(o_auto).all()
    assert rel_err(o_s28, o_auto) < TOL_BF16
    sub = slice(U - 2, U)
    st2 = cabi.LayerStore(2, D, G, R, n_quant, torch.bfloat16, "cuda")
    cabi.load_state(st2, k[sub], v[sub], n_quant)
    o_f32 = st2.attention(q[sub].contiguous(), n_rep=n_rep, path=cabi.ATTN_FP32, out_dtype=torch.float32)
    print(f"[cfg3 full size] tensor-core vs fp32 kernel {rel_err(o_auto[sub], o_f32):.2e}")
    assert rel_err(o_auto[sub], o_f32) < TOL_BF16
    u = 5
    kk, vv = k[u:u + 1].cpu().reshape(1, 1, T, D), v[u:u + 1].cpu().reshape(1, 1, T, D)
    ref = ko.kivi_decode_attention(q[u:u + 1].cpu().reshape(1, n_rep, D), kk, vv, n_quant, G, "half_away",
                                   dtype=torch.float64).float().reshape(1, n_rep, D)
    e_row, e_el = rel_err(o_auto[u:u + 1], ref), elem_err(o_auto[u:u + 1], ref)
    print(f"[cfg3 full size] unit {u} vs oracle: rel err {e_row:.2e}, element-wise {e_el:.2e}")
    assert e_row < TOL_BF16


def test_full_size_config4_prefill_properties(cabi):
    """Bulk prefill at the benchmark's full size (256 units, 8192 tokens, bf16):
    the round trip through the packed store stays within half a quantization
    step of the input for every element (step = the stored scale of its group),
    ring tokens come back exactly, and two sampled units equal the CPU oracle bit
    for bit (codes through the dequantized values, scales and zeros directly)."""
    U, S, D, G, R = 256, 8192, 128, 32, 128
    g = torch.Generator(device="cuda").manual_seed(77)
    k = torch.empty(U, S, D, device="cuda", dtype=torch.bfloat16)
    v = torch.empty(U, S, D, device="cuda", dtype=torch.bfloat16)
    for u0 in range(0, U, 64):
        k[u0:u0 + 64] = torch.randn(64, S, D, device="cuda", generator=g).to(torch.bfloat16)
        v[u0:u0 + 64] = torch.randn(64, S, D, device="cuda", generator=g).to(torch.bfloat16)
    k[:, :, 9] *= 10.0
    st = cabi.LayerStore(U, D, G, R, S, torch.bfloat16, "cuda")
    st.update(k, v)
    n_flush, ql, rl = cabi.cache_plan(0, 0, S, G, R)
    assert (st.quant_len, st.res_len) == (ql, rl) == (S - 96, 96)
    ng = ql // G
    for name, x, by_token in (("k", k, False), ("v", v, True)):
        served = st.materialize()[1 if by_token else 0]                     # fp32 [U, S, D]
        assert torch.equal(served[:, ql:], x[:, ql:].float()), f"{name}: ring tokens must come back exactly"
        if by_token:        # scale of (token t, channel group gd); stored rows are permuted inside 32-token blocks
            rows = st.v_scales[:, :ql].reshape(U, ng, 2, 4, 4, D // G).permute(0, 1, 2, 4, 3, 5).reshape(U, ql, D // G)
            step = rows.repeat_interleave(G, dim=2)
        else:               # scale of (group g, channel d)
            step = st.k_scales[:, :ng].repeat_interleave(G, dim=1)
        worst = 0.0
        for u0 in range(0, U, 32):                                           # bounded temporaries
            err = (served[u0:u0 + 32, :ql] - x[u0:u0 + 32, :ql].float()).abs()
            bound = step[u0:u0 + 32] * 0.5 * (1 + 1e-5) + 1e-30
            assert bool((err <= bound).all()), f"{name}: round trip off by more than half a step"
            worst = max(worst, float((err / step[u0:u0 + 32]).max()))
        print(f"[cfg4 full size] {name}: worst |error| / step = {worst:.4f}")
        del served, step
    # two units against the oracle
    for u in (3, 200):
        oc = ko.OracleCache(D, G, R, rounding="half_away")
        ku, vu = k[u].float().cpu().reshape(1, 1, S, D), v[u].float().cpu().reshape(1, 1, S, D)
        oc.append(ku, vu)
        sk, sv = oc.served()
        one = cabi.LayerStore(1, D, G, R, S, torch.bfloat16, "cuda")
        one.update(k[u:u + 1], v[u:u + 1])
        gk, gv = one.materialize()
        assert torch.equal(gk.cpu(), sk.reshape(1, S, D)) and torch.equal(gv.cpu(), sv.reshape(1, S, D))
        assert torch.equal(one.k_scales[0, :ng].cpu(), torch.stack(oc.k_scales, dim=2).reshape(ng, D))
        assert torch.equal(st.k_scales[u, :ng].cpu(), one.k_scales[0, :ng].cpu())
        assert torch.equal(st.v_codes[u, :ql].cpu(), one.v_codes[0, :ql].cpu())


@pytest.mark.parametrize("dtype,path", [(torch.bfloat16, "mma"), (torch.float32, "fp32")])
def test_attention_lse_combines_token_shards(cabi, dtype, path):
    """kivi_decode_attention_lse: the log-sum-exp equals the oracle's, and two
    stores holding disjoint token ranges of the same sequences (sequence
    sharding on one GPU) combine into the single-store result."""
    from intel_kivi_hybrid_b200.parallel import merge_token_shards
    B, H, n_rep, D, G, R = 1, 4, 4, 128, 32, 128
    n_quant, n_res, n1 = 1024, 77, 384
    T, U = n_quant + n_res, B * H
    K = ko.make_keys(B, H, T, D, seed=13)
    V = ko.make_values(B, H, T, D, seed=13)
    q = ko.make_queries(B, H * n_rep, D, seed=13)
    if dtype == torch.bfloat16:
        K, V, q = K.bfloat16().float(), V.bfloat16().float(), q.bfloat16().float()
    kc, vc = units(K).cuda().to(dtype), units(V).cuda().to(dtype)
    qd = q.reshape(U, n_rep, D).cuda().to(dtype)
    p = cabi.ATTN_MMA if path == "mma" else cabi.ATTN_FP32
    whole = cabi.LayerStore(U, D, G, R, n_quant, dtype, "cuda")
    cabi.load_state(whole, kc, vc, n_quant)
    out_w, lse_w = whole.attention_lse(qd, n_rep=n_rep, path=p, out_dtype=torch.float32)
    assert torch.equal(out_w, whole.attention(qd, n_rep=n_rep, path=p, out_dtype=torch.float32))
    # oracle log-sum-exp over the served cache
    kd, vd = whole.materialize()
    s = torch.einsum("uhd,utd->uht", qd.double().cpu(), kd.double().cpu()) * D ** -0.5
    assert torch.allclose(lse_w.cpu().double(), torch.logsumexp(s, -1), atol=2e-3 if dtype == torch.bfloat16 else 2e-5)
    # many pieces per unit: the fold done by a whole CTA per row gives the same log-sum-exp
    out_m, lse_m = whole.attention_lse(qd, n_rep=n_rep, path=p, out_dtype=torch.float32, num_splits=24)
    assert torch.allclose(lse_m, lse_w, atol=1e-5 if dtype == torch.float32 else 1e-4)
    assert rel_err(out_m, out_w) < (TOL_F32 if dtype == torch.float32 else TOL_BF16)
    # shard 0: the first n1 tokens, all quantized; shard 1: the rest with the ring
    s0 = cabi.LayerStore(U, D, G, R, n1, dtype, "cuda")
    cabi.load_state(s0, kc[:, :n1], vc[:, :n1], n1)
    s1 = cabi.LayerStore(U, D, G, R, n_quant - n1, dtype, "cuda")
    cabi.load_state(s1, kc[:, n1:], vc[:, n1:], n_quant - n1)
    o0, l0 = s0.attention_lse(qd, n_rep=n_rep, path=p, out_dtype=torch.float32)
    o1, l1 = s1.attention_lse(qd, n_rep=n_rep, path=p, out_dtype=torch.float32)
    merged = merge_token_shards(torch.stack([o0, o1]), torch.stack([l0, l1]))
    tol = TOL_BF16 if dtype == torch.bfloat16 else TOL_F32
    assert rel_err(merged, out_w) < tol
    ref = ko.kivi_decode_attention(q, K, V, n_quant, G, "half_away", dtype=torch.float64).float().reshape(U, n_rep, D)
    assert rel_err(merged, ref) < tol
    with pytest.raises(RuntimeError, match="empty cache"):
        cabi.LayerStore(U, D, G, R, 64, dtype, "cuda").attention_lse(qd, n_rep=n_rep)


@pytest.mark.parametrize("chunks,direct", [(1, True), (1, False), (2, False), (3, False)])
def test_decode_step_from_host_equals_update_then_attention(cabi, chunks, direct):
    """kivi_decode_step_host: pinned host q / new token in, pinned host output back.
    Over 40 steps (one flush inside) the counters, the packed store and the ring
    must end up bit-identical to update() + attention() called separately; the
    outputs are bit-identical with one chunk (same split plan) and within the
    tolerance of the oracle with several."""
    B, Hkv, n_rep, D, G, R = 2, 4, 4, 128, 32, 128
    U, T0, steps = B * Hkv, 700, 40
    K = ko.make_keys(B, Hkv, T0 + steps, D, seed=31).to(torch.bfloat16)
    V = ko.make_values(B, Hkv, T0 + steps, D, seed=31).to(torch.bfloat16)
    Kc, Vc = units(K).cuda(), units(V).cuda()
    a = cabi.LayerStore(U, D, G, R, 1024, torch.bfloat16, "cuda")
    b = cabi.LayerStore(U, D, G, R, 1024, torch.bfloat16, "cuda")
    a.update(Kc[:, :T0], Vc[:, :T0]); b.update(Kc[:, :T0], Vc[:, :T0])
    h_q = torch.empty(U, n_rep, D, dtype=torch.bfloat16).pin_memory()
    h_k = torch.empty(U, D, dtype=torch.bfloat16).pin_memory()
    h_v = torch.empty(U, D, dtype=torch.bfloat16).pin_memory()
    h_out = torch.empty(U, n_rep, D, dtype=torch.float32).pin_memory()
    worst = 0.0
    for t in range(T0, T0 + steps):
        q = ko.make_queries(B, Hkv * n_rep, D, seed=t).to(torch.bfloat16)
        h_q.copy_(q.reshape(U, n_rep, D)); h_k.copy_(units(K)[:, t]); h_v.copy_(units(V)[:, t])
        a.decode_step_host(h_q, h_k, h_v, h_out, n_rep, chunks=chunks, direct=direct)
        b.update(Kc[:, t:t + 1], Vc[:, t:t + 1])
        ref_out = b.attention(q.reshape(U, n_rep, D).cuda(), n_rep=n_rep, out_dtype=torch.float32)
        torch.cuda.synchronize()
        assert (a.quant_len, a.res_start, a.res_len) == (b.quant_len, b.res_start, b.res_len)
        if chunks == 1:
            assert torch.equal(h_out, ref_out.cpu())
        else:
            assert rel_err(h_out, ref_out) < TOL_BF16
        if t % 13 == 0:
            ref = ko.kivi_decode_attention(q, K[:, :, :t + 1], V[:, :, :t + 1], a.quant_len, G, "half_away", dtype=torch.float64)
            worst = max(worst, rel_err(h_out, ref.float().reshape(U, n_rep, D)))
    assert a.quant_len == 640 and worst < TOL_BF16
    for name in ("k_codes", "k_scales", "k_zeros", "v_codes", "v_scales", "v_zeros", "k_res", "v_res"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    assert cabi.device_fault() == 0
    with pytest.raises(RuntimeError, match="pinned"):
        a.decode_step_host(h_q.clone(), h_k, h_v, h_out, n_rep)


def test_tensor_core_keeps_enough_bits_for_subnormal_codes(cabi):
    """The tensor-core kernel feeds codes as fp16 subnormals; the MMA aligns its
    addends on their exponent fields and truncates a fixed distance below the
    largest.  The kernel's placement of the codes (no code lower than bits 2-3 of
    its half) leaves 20 bits if the unit keeps 26 below the largest addend's
    leading bit, i.e. still resolves 2^-25 next to 1."""
    bits = cabi.mma_alignment_bits()
    print(f"[tensor core] 1 + 2^-k - 1 is exact up to k = {bits}")
    assert bits >= 24


@pytest.mark.parametrize("D,G,R,ring,new,shift,strided", [
    (128, 32, 128, torch.bfloat16, torch.bfloat16, 0, False), (64, 16, 96, torch.float32, torch.float32, 0, True),
    (128, 32, 64, torch.float32, torch.bfloat16, 0, True), (64, 32, 128, torch.bfloat16, torch.float32, 0, False),
    (12, 4, 8, torch.float32, torch.float32, 0, False),                     # head_dim not a multiple of eight
    (128, 32, 128, torch.bfloat16, torch.bfloat16, 1, False),               # new tensor off the 16-byte grid
])
def test_ring_append_keeps_the_window(cabi, D, G, R, ring, new, shift, strided):
    """The window after chunks of every length (single tokens, wrap-around, bulk) is
    the last res_len tokens, bit for bit (fp32 to a bf16 ring: rounded to nearest)."""
    U, g = 3, torch.Generator(device="cuda").manual_seed(D + R)
    T = 6 * R
    st = cabi.LayerStore(U, D, G, R, T, ring, "cuda")
    wide = D + 8 if strided else D
    flat = [torch.randn(U * T * wide + shift, generator=g, device="cuda").to(new)[shift:].view(U, T, wide)[..., :D] for _ in range(2)]
    t = 0
    for n in (1, 2, R // 2 + 1, 1, R - 1, 3, 1, R + G + 1, 1):
        st.update(flat[0][:, t:t + n], flat[1][:, t:t + n])
        t += n
        assert st.quant_len + st.res_len == t
        idx = (torch.arange(st.res_len, device="cuda") + st.res_start) % R
        for x, buf in ((flat[0], st.k_res), (flat[1], st.v_res)):
            assert torch.equal(buf[:, idx], x[:, t - st.res_len:t].to(ring)), (n, t)


@pytest.mark.parametrize("D,G,n_rep,n_quant,n_res,res_start,dtype", [
    (64, 4, 1, 36, 0, 0, torch.float32),             # groups of four tokens: one of eight token quads in use
    (128, 8, 3, 8 * 9, 5, 60, torch.float32), (64, 16, 2, 16 * 33, 31, 40, torch.bfloat16),
    (64, 64, 8, 64 * 5, 33, 0, torch.float32),       # two runs of 32 tokens per group
    (128, 128, 7, 128 * 3, 64, 1, torch.bfloat16), (128, 32, 5, 32 * 17, 1, 63, torch.float32),
    (128, 32, 1, 0, 64, 10, torch.float32),          # nothing quantized
    (64, 32, 6, 32, 0, 0, torch.bfloat16),           # one group, empty ring
    (32, 8, 4, 64, 20, 50, torch.float32), (256, 64, 2, 128, 20, 50, torch.float32),      # other head_dims: generic kernel
])
def test_attention_fp32_kernels_at_their_edges(cabi, D, G, n_rep, n_quant, n_res, res_start, dtype):
    """fp32-arithmetic kernels against 64 bits on the cache's own dequantized keys and
    values.  Bound 1e-5 of the row's largest element (fp32 activations): sums of at
    most n_quant + n_res + D products in fp32, 2^-24 * sqrt(600) = 1.5e-6 per rounding chain."""
    U, g = 3, torch.Generator(device="cuda").manual_seed(D * G + n_rep)
    T = n_quant + n_res
    st = cabi.LayerStore(U, D, G, 128, max(n_quant, G), dtype, "cuda")
    k, v = (torch.randn(U, T, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    cabi.load_state(st, k, v, n_quant)
    st.k_res, st.v_res = (torch.roll(x, res_start, dims=1).contiguous() for x in (st.k_res, st.v_res))
    st.c.k_res, st.c.v_res, st.res_start = st.k_res.data_ptr(), st.v_res.data_ptr(), res_start
    q = torch.randn(U, n_rep, D, generator=g, device="cuda").to(dtype)
    kd, vd = st.materialize()
    w = torch.softmax(q.double() @ kd.double().transpose(1, 2) * D ** -0.5, dim=-1)
    ref = w @ vd.double()
    for splits in (0, 1, 3):
        out = st.attention(q, n_rep=n_rep, path=cabi.ATTN_FP32, out_dtype=torch.float32, num_splits=splits)
        err = ((out.double() - ref).abs().amax(-1) / ref.abs().amax(-1)).max().item()
        assert err < 1e-5, (splits, err)


@pytest.mark.parametrize("D,G,n_rep,n_res,res_start,ring", [
    (64, 32, 3, 20, 120, torch.float32), (64, 16, 8, 128, 127, torch.bfloat16),
    (128, 32, 1, 33, 96, torch.bfloat16), (128, 128, 4, 100, 101, torch.float32), (128, 8, 8, 128, 65, torch.float32)])
def test_attention_fp32_tile_kernel_across_the_end_of_the_ring(cabi, D, G, n_rep, n_res, res_start, ring):
    """The window lies across the end of a ring of 128 slots, in each kind of the tile
    kernel's ring code: both head_dims, both ring types, one and several heads.
    Bound as in the test of the kernels' edges above."""
    U, R, n_quant = 3, 128, 2 * G
    assert res_start + n_res > R
    g = torch.Generator(device="cuda").manual_seed(D + G + n_rep)
    st = cabi.LayerStore(U, D, G, R, n_quant, ring, "cuda")
    k, v = (torch.randn(U, n_quant + n_res, D, generator=g, device="cuda").to(ring) for _ in range(2))
    cabi.load_state(st, k, v, n_quant)
    for buf in (st.k_res, st.v_res):
        buf.copy_(torch.roll(buf, res_start, dims=1))
    st.res_start = res_start
    q = torch.randn(U, n_rep, D, generator=g, device="cuda")
    kd, vd = st.materialize()
    assert torch.equal(kd[:, n_quant:], k[:, n_quant:].float())
    ref = torch.softmax(q.double() @ kd.double().transpose(1, 2) * D ** -0.5, dim=-1) @ vd.double()
    assert rel_err(st.attention(q, n_rep=n_rep), ref) < TOL_F32


@pytest.mark.parametrize("D,G,n_rep,path,dtype", [
    (64, 32, 1, "fp32", torch.float32), (64, 64, 8, "fp32", torch.bfloat16), (128, 32, 4, "fp32", torch.float32), (128, 128, 7, "fp32", torch.float32),
    (128, 32, 1, "mma", torch.bfloat16), (128, 32, 3, "mma", torch.bfloat16), (128, 32, 8, "mma", torch.bfloat16)])
def test_fold_in_a_cluster_gives_the_bits_of_the_fold_kernel(cabi, D, G, n_rep, path, dtype):
    """Few units fold inside clusters of the attention kernel, many leave it to the fold
    kernel; a unit's output and log-sum-exp do not depend on which, bit for bit, for
    every piece count a cluster takes."""
    few, many, n_quant, n_res = 3, 160, 8 * G, 40             # 160 units: more CTAs than SMs whatever the cut
    g = torch.Generator(device="cuda").manual_seed(D + n_rep)
    k, v = (torch.randn(few, n_quant + n_res, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    q = torch.randn(few, n_rep, D, generator=g, device="cuda").to(dtype)
    kernel = cabi.ATTN_FP32 if path == "fp32" else cabi.ATTN_MMA
    for res in (n_res, 0):
        outs = []
        for U in (few, many):
            st = cabi.LayerStore(U, D, G, 128, n_quant, dtype, "cuda")
            pad = lambda x: torch.cat([x, x[:1].expand(U - few, *x.shape[1:])])
            cabi.load_state(st, pad(k)[:, :n_quant + res], pad(v)[:, :n_quant + res], n_quant)
            per = []
            for pieces in range(1, 8):
                out, lse = st.attention_lse(pad(q).contiguous(), n_rep=n_rep, num_splits=pieces, path=kernel, out_dtype=torch.float32)
                launches = cabi.lib.kivi_last_launch_count()
                assert launches == (1 if U == few else 2), (U, pieces, launches)
                per.append((out[:few], lse[:few]))
            outs.append(per)
        for (o1, l1), (o2, l2) in zip(*outs):
            assert torch.equal(o1, o2) and torch.equal(l1, l2)


@pytest.mark.parametrize("what", ["tiny", "huge", "mixed", "negative", "k_inf", "k_nan", "v_inf", "v_nan", "q_nan"])
@pytest.mark.parametrize("tokens,n_rep", [(32, 1), (96, 4), (288, 3), (320, 8)])
def test_attention_mma_at_the_edges_of_its_fixed_point_operands(cabi, what, tokens, n_rep):
    """q*s and p*s go to the tensor cores as fixed-point numbers of the largest of a stage
    (two groups; one at an odd end): scales of any size, of sizes far apart and negative
    value scales give what the fp32 kernel gives; infinities and NaN come out where they do there.
    A weight is off by 2^-16 of the stage's largest at most and its code is 3 at most; all 64
    of a stage wrong the same way would be 64 * 3 * 2^-16 = 2.9e-3 of the largest value."""
    U = 5
    st = cabi.LayerStore(U, 128, 32, 128, tokens, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(tokens + n_rep)
    for n in ("k_codes", "v_codes"):
        getattr(st, n).random_(0, 256, generator=g)
    for n, lo, hi in (("k_scales", 0.3, 1.2), ("v_scales", 0.3, 1.2), ("k_zeros", -2.0, -0.5), ("v_zeros", -2.0, -0.5)):
        getattr(st, n).uniform_(lo, hi, generator=g)
    st.quant_len = tokens
    q = torch.randn(U, n_rep, 128, generator=g, device="cuda").bfloat16()
    if what in ("tiny", "huge"):
        f = 1e-30 if what == "tiny" else 1e30
        for n in ("v_scales", "v_zeros"):
            getattr(st, n).mul_(f)
        for n in ("k_scales", "k_zeros"):
            getattr(st, n).mul_(f)
        q = (q.float() / f).bfloat16()
    elif what == "mixed":                                       # one channel and one token a million times the others
        st.k_scales[:, :, 7] *= 1e6
        q[:, :, 7] *= 1e-6
        st.v_scales.view(U, -1)[:, 5] *= 1e6
    elif what == "negative":
        st.v_scales.view(U, -1)[:, 11] *= -1
        st.k_scales[:, 0, 3] *= -1
    elif what in ("k_inf", "k_nan"):
        st.k_scales[2, -1, 77] = float(what[2:])
    elif what in ("v_inf", "v_nan"):
        st.v_scales.view(U, -1)[2, 13] = float(what[2:])
    elif what == "q_nan":
        q[3, 0, 100] = float("nan")
    got, want = (st.attention(q, n_rep=n_rep, path=p, out_dtype=torch.float32) for p in (cabi.ATTN_MMA, cabi.ATTN_FP32))
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert want.isfinite().any() and cabi.device_fault() == 0
    if what in ("tiny", "huge", "mixed", "negative"):
        assert want.isfinite().all()
    ok = want.isfinite()
    size = (st.v_scales.abs().nan_to_num(0, 0, 0).max() * 3 + st.v_zeros.abs().max()).item()
    assert ((got - want)[ok].abs().max() / size).item() < 2.9e-3


@pytest.mark.parametrize("loud", ["channel group", "token group"])
@pytest.mark.parametrize("dtype,n_rep", [(torch.bfloat16, 1), (torch.bfloat16, 2), (torch.bfloat16, 4), (torch.bfloat16, 8), (torch.float32, 4)])
@pytest.mark.parametrize("n_quant,n_res", [(96, 5), (1056, 0)])
def test_attention_beside_a_louder_neighbour(cabi, n_quant, n_res, dtype, n_rep, loud):
    """Values of one channel group, or keys of every other token group (far below the others in
    the softmax), thousands of times larger than their neighbours: every channel group of a row
    keeps the tolerance against its own largest output.  (A weight is off by less than 2^-16 of the
    largest of its own sums: 64 of a stage, three at most of a code, as independent roundings
    3 * 8 * 2^-16 = 3.7e-4 of the largest weight, a fifth of the bf16 tolerance; fp32 2^-15 of that.)"""
    B, Hkv, D, G, T = 1, 3, 128, 32, n_quant + n_res
    K, V = ko.make_keys(B, Hkv, T, D, 23), ko.make_values(B, Hkv, T, D, 23)
    q = ko.make_queries(B, Hkv * n_rep, D, 23)
    if loud == "channel group":
        V[..., 32:64] *= 2.0 ** 14
    else:
        q[..., 0] = 3.0
        K[..., 0] = 0.0
        for t in range(0, n_quant, 2 * G):
            K[:, :, t:t + G] *= 2.0 ** 14
            K[:, :, t:t + G, 0] = -100.0 * 2.0 ** 14
    K, V, q = K.to(dtype), V.to(dtype), q.to(dtype)
    st = cabi.LayerStore(B * Hkv, D, G, 128, n_quant, dtype, "cuda")
    cabi.load_state(st, units(K).cuda(), units(V).cuda(), n_quant)
    out = st.attention(q.cuda(), n_rep=n_rep, out_dtype=torch.float32)
    ref = ko.kivi_decode_attention(q, K, V, n_quant, G, "half_away", dtype=torch.float64)
    err = rel_err(out.view(-1, 4, 32), ref.view(-1, 4, 32).float())
    print(f"[attn beside a louder {loud} {dtype} heads={n_rep} q={n_quant}] rel err {err:.2e}")
    assert err < (TOL_BF16 if dtype == torch.bfloat16 else TOL_F32) and cabi.device_fault() == 0


@pytest.mark.parametrize("n_quant,n_res,n_rep,splits", [(1024, 0, 3, 1), (1056, 77, 4, 0), (1312, 128, 5, 7), (4064, 200, 8, 0), (2080, 1, 4, 65)])
def test_attention_fp32_queries_on_the_tensor_cores(cabi, n_quant, n_res, n_rep, splits):
    """From three heads and 1024 tokens on fp32 queries are served there: whole and odd
    stages, one to 65 pieces, one and two head blocks, several ring parts."""
    assert cabi.attention_plan(2, n_quant, n_res, n_rep=n_rep, q_dtype=cabi.F32, num_splits=splits)[0]
    err, oerr, _, _ = _attention_case(cabi, 1, 2, n_rep, 128, 32, 256, n_quant, n_res, torch.float32, 3, cabi.ATTN_AUTO, num_splits=splits)
    print(f"[attn fp32 on tensor cores q={n_quant} r={n_res} heads={n_rep}] rel err {err:.2e} (fp32 oracle: {oerr:.2e})")
    assert err < TOL_F32 and cabi.device_fault() == 0


@pytest.mark.parametrize("what", ["tiny", "huge", "mixed", "negative", "k_inf", "v_nan", "q_nan"])
def test_attention_fp32_queries_at_the_edges_of_fixed_point(cabi, what):
    """As for bf16 queries above, with the longer operands: a weight is off by 2^-30 of the
    stage's largest at most and a score by that of 128 channels, so the fp32 tolerance holds."""
    U, tokens, n_rep = 3, 1056, 4
    st = cabi.LayerStore(U, 128, 32, 128, tokens, torch.float32, "cuda")
    g = torch.Generator(device="cuda").manual_seed(17)
    for n in ("k_codes", "v_codes"):
        getattr(st, n).random_(0, 256, generator=g)
    for n, lo, hi in (("k_scales", 0.3, 1.2), ("v_scales", 0.3, 1.2), ("k_zeros", -2.0, -0.5), ("v_zeros", -2.0, -0.5)):
        getattr(st, n).uniform_(lo, hi, generator=g)
    st.quant_len = tokens
    q = torch.randn(U, n_rep, 128, generator=g, device="cuda")
    if what in ("tiny", "huge"):
        f = 1e-30 if what == "tiny" else 1e30
        for n in ("v_scales", "v_zeros", "k_scales", "k_zeros"):
            getattr(st, n).mul_(f)
        q /= f
    elif what == "mixed":
        st.k_scales[:, :, 7] *= 1e4
        st.k_zeros[:, :, 7] *= 1e4
        q[:, :, 7] *= 1e-4
        st.v_scales.view(U, -1)[:, 5] *= 1e4
    elif what == "negative":
        st.v_scales.view(U, -1)[:, 11] *= -1
        st.k_scales[:, 0, 3] *= -1
    elif what == "k_inf":
        st.k_scales[2, -1, 77] = float("inf")
    elif what == "v_nan":
        st.v_scales.view(U, -1)[2, 13] = float("nan")
    elif what == "q_nan":
        q[1, 0, 100] = float("nan")
    got, want = (st.attention(q, n_rep=n_rep, path=p) for p in (cabi.ATTN_AUTO, cabi.ATTN_FP32))
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    ok = want.isfinite()
    assert ok.any() and cabi.device_fault() == 0
    size = want[ok].abs().max()
    assert ((got - want)[ok].abs().max() / size).item() < 2 * TOL_F32          # both are within it of the exact result


def test_fp32_queries_keep_to_the_scratch_they_are_given(cabi):
    """What the CUDA-core kernel's partials (one ring part at most) fit is served, by the
    tensor-core kernel with fewer pieces or by that kernel itself; what they do not fit is refused."""
    U, T, n_rep, D = 40, 4096, 4, 128
    st = cabi.LayerStore(U, D, 32, 1024, T, torch.float32, "cuda")
    k, v = (torch.randn(U, T + 1000, D, device="cuda") for _ in range(2))
    cabi.load_state(st, k, v, T)
    q = torch.randn(U, n_rep, D, device="cuda")
    want = st.attention(q, n_rep=n_rep, path=cabi.ATTN_FP32)
    row = U * n_rep * (D + 2) * 4
    # the least an automatic count of the CUDA-core kernel needs: its plan or about eight CTAs per SM
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    least = min(cabi.attention_plan(U, T, 1000, n_rep=n_rep, q_dtype=cabi.F32)[1], -(-8 * sms // U), T // 32 // 4) + 1
    # (pieces asked for, partials of a row the workspace holds); 1000 window tokens are eight ring parts
    for pieces, ring, served in ((0, 40, True), (0, least, True), (0, least - 1, False), (1, 2, True), (1, 9, True), (5, 6, True), (5, 5, False)):
        out = torch.empty_like(q)
        ws = torch.empty(row * ring, dtype=torch.uint8, device="cuda")
        rc = cabi.lib.kivi_decode_attention(ctypes.byref(st.c), T, st.res_start, st.res_len, q.data_ptr(), cabi.F32, out.data_ptr(), cabi.F32, n_rep, 0.0,
                                            ws.data_ptr(), ws.numel(), pieces, cabi.ATTN_AUTO, torch.cuda.current_stream().cuda_stream)
        assert (rc == 0) == served, (pieces, ring, cabi.lib.kivi_last_error())
        if served:
            assert rel_err(out, want.cpu()) < 2 * TOL_F32, (pieces, ring)


@pytest.mark.parametrize("D,dtype,U,n_rep", [(128, torch.bfloat16, 8, 4), (64, torch.float32, 12, 1), (128, torch.bfloat16, 200, 1), (32, torch.float32, 2, 2)])
def test_queued_steps_equal_synchronised_steps(cabi, D, dtype, U, n_rep):
    """Launches overlap the kernels before them in their stream: append, flush,
    attention and sampling of 70 steps queued without a pause (flushes among them) leave the
    same bits as the same steps with the GPU idle before each call."""
    G = 8 if D == 32 else 32                                   # (head_dim 32: the generic kernels)
    steps, T0 = 70, 200
    g = torch.Generator(device="cuda").manual_seed(U)
    k, v = (torch.randn(U, T0 + steps, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    q = torch.randn(steps, U, n_rep, D, generator=g, device="cuda").to(dtype)
    results = []
    for queued in (True, False):
        st = cabi.LayerStore(U, D, G, 128, 512, dtype, "cuda")
        wait = (lambda: None) if queued else torch.cuda.synchronize
        outs, ids = [], []
        torch.cuda.synchronize()
        st.update(k[:, :T0], v[:, :T0])
        for i in range(steps):
            wait()
            st.update(k[:, T0 + i:T0 + i + 1], v[:, T0 + i:T0 + i + 1])
            wait()
            outs.append(st.attention(q[i], n_rep=n_rep))
            wait()
            outs.append(st.attention(q[i], n_rep=n_rep, num_splits=1))
            wait()
            ids.append(cabi.sample_tokens(outs[-1].view(U, -1), 1.0, 5, True, seed=i))
        torch.cuda.synchronize()
        results.append((torch.stack(outs), torch.stack(ids), *st.materialize(), st.k_res.clone(), st.v_res.clone()))
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert cabi.device_fault() == 0


_TWO_THREADS_CPP = r"""
#include <atomic>
#include <thread>
#include "kivi_cuda.h"
extern "C" void together(const kivi_layer* const* layers, const void* q, void* const* outs, void* const* ws, size_t ws_bytes, int64_t tokens,
                         int n_rep, int* rc) {
    std::atomic<int> ready{0};
    auto work = [&](int i) {
        ready.fetch_add(1);
        while (ready.load() < 2) {}
        rc[i] = kivi_decode_attention(layers[i], tokens, 0, 0, q, KIVI_F32, outs[i], KIVI_F32, n_rep, 0.0f, ws[i], ws_bytes, 0, KIVI_ATTN_FP32, nullptr);
    };
    std::thread a(work, 0), b(work, 1);
    a.join(); b.join();
}
"""
_TWO_THREADS = r"""
import ctypes, sys, torch
sys.path.insert(0, sys.argv[1])
from intel_kivi_hybrid_b200 import cabi
together = ctypes.CDLL(sys.argv[2]).together
D, T, U, failed = 128, 256, 2, []
stores = [cabi.LayerStore(U, D, G, 128, T, torch.float32, "cuda") for G in (128, 64)]
for st in stores:
    cabi.load_state(st, torch.randn(U, T, D, device="cuda"), torch.randn(U, T, D, device="cuda"), T)
torch.cuda.synchronize()
vp = ctypes.c_void_p
for n_rep in range(1, 9):                       # each head count is a kernel of its own, met here for the first time
    q = torch.randn(U, n_rep, D, device="cuda")
    outs, ws, rc = [torch.empty_like(q) for _ in stores], [st.workspace(n_rep) for st in stores], (ctypes.c_int * 2)()
    torch.cuda.synchronize()
    two = lambda p: (vp * 2)(*p)
    together(two([ctypes.addressof(st.c) for st in stores]), vp(q.data_ptr()), two([o.data_ptr() for o in outs]), two([w.data_ptr() for w in ws]),
             ctypes.c_size_t(ws[0].numel()), ctypes.c_int64(T), n_rep, rc)
    failed += [(n_rep, st.G, "together") for st, c in zip(stores, rc) if c]
    for st in stores:
        try:
            st.attention(q, n_rep=n_rep)
        except RuntimeError as e:
            failed.append((n_rep, st.G, str(e)))
torch.cuda.synchronize()
print("failed:", failed)
sys.exit(1 if failed else 0)
"""


def test_first_fp32_attention_calls_from_two_threads(tmp_path):
    """Groups of 64 and of 128 tokens need different amounts of shared memory of the same
    kernel: two host threads that launch it for the first time together must not leave it
    with the smaller limit.  A process of its own: a kernel is met for the first time once."""
    from intel_kivi_hybrid_b200 import _build
    (tmp_path / "two.cpp").write_text(_TWO_THREADS_CPP)
    (tmp_path / "two.py").write_text(_TWO_THREADS)
    lib = str(tmp_path / "two.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I" + os.path.join(_build.ROOT, "include"), str(tmp_path / "two.cpp"),
                    "-o", lib, "-L" + _build.PKG, "-l:libkivi_cuda.so", "-Wl,-rpath," + _build.PKG], check=True)
    p = subprocess.run([sys.executable, str(tmp_path / "two.py"), _build.ROOT, lib], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
