"""Each sm_100a kernel against the fp32 PyTorch definition of the same op (small shapes,
odd sizes, tails).  Tolerances: bf16 outputs 2e-2 relative to the row scale, fp32 1e-4."""
import math

import pytest
import torch

from coffin_b200.oracle import ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def K():
    from coffin_b200.ops import kernels
    return kernels


def close(got, ref, tol=2e-2):
    got, ref = got.float().cpu(), ref.float().cpu()
    scale = ref.abs().max().clamp_min(1e-6)
    err = (got - ref).abs().max() / scale
    assert torch.isfinite(got).all()
    assert err < tol, f"relative error {err:.4g} (scale {scale:.4g})"


def bf(*shape, s=1.0, seed=0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * s).to(torch.bfloat16)


@pytest.mark.parametrize("M,N", [(300, 520), (257, 2560), (1000, 5120), (256, 1000), (2048, 3072)])
def test_rmsnorm_many_rows(M, N):
    """Prefill-sized calls run one warp per row with the row in registers (chunks per lane 4 / 8 / 12 / 20)."""
    k = K()
    x, add = bf(M, N, seed=5), bf(M, N, seed=6)
    gain = (1 + 0.1 * torch.randn(N)).float()
    canary = torch.full((M + 1, N), 3.0, dtype=torch.bfloat16, device=DEV)
    out = k.rmsnorm(x.to(DEV), gain.to(DEV), 1e-6, out=canary[:M])
    close(out, O.rms_norm(x, gain))
    assert bool((canary[M] == 3.0).all())
    res = x.to(DEV)
    out = k.rmsnorm(res, gain.to(DEV), 1e-6, add=add.to(DEV), res_out=res)      # in place, as the model does
    s, n = O.add_rms_norm(x, add, gain)
    close(res, s)
    close(out, n)
    # int8 rows + scales straight from the norm kernel == quantising its bf16 output afterwards
    q8 = torch.empty(M, N, dtype=torch.int8, device=DEV)
    s8 = torch.empty(M, dtype=torch.float32, device=DEV)
    k.rmsnorm(x.to(DEV), gain.to(DEV), 1e-6, quant=(q8, s8))
    qr, sr = k.quant_rows(k.rmsnorm(x.to(DEV), gain.to(DEV), 1e-6))
    assert torch.equal(q8, qr) and torch.equal(s8, sr)
    # the vectorised quantiser against its definition (SwiGLU form included)
    gu = bf(M, 2 * N, seed=8)
    for sw, src in ((False, x), (True, gu)):
        qv, sv = k.quant_rows(src.to(DEV), swiglu=sw)
        v = O.silu_mul(src[:, :N], src[:, N:]).to(torch.bfloat16).float() if sw else src.float()
        sc = v.abs().amax(-1).clamp_min(1e-8) / 127
        ref = torch.clamp(torch.round(v / sc[:, None]), -127, 127)
        assert (sv.cpu() - sc).abs().max() <= 1e-6 * sc.max() + 1e-12
        assert (qv.cpu().float() - ref).abs().max() <= 1      # a value on a rounding boundary may land either side


def test_rowwise_kernels():
    k = K()
    x, add = bf(5, 520, seed=1), bf(5, 520, seed=2)
    gain = (1 + 0.1 * torch.randn(520)).float()
    out = k.rmsnorm(x.to(DEV), gain.to(DEV), 1e-6)
    close(out, O.rms_norm(x, gain))
    res = torch.empty_like(x, device=DEV)
    out = k.rmsnorm(x.to(DEV), gain.to(DEV), 1e-6, add=add.to(DEV), res_out=res)
    s, n = O.add_rms_norm(x, add, gain)
    close(res, s)
    close(out, n)
    gu = bf(7, 2 * 264, seed=3)
    close(k.swiglu(gu.to(DEV)), O.silu_mul(gu[:, :264], gu[:, 264:]))
    logits = torch.randn(3, 4099)
    logits[1, 77] = logits[1, 4000] = 50.0
    assert k.argmax(logits.to(DEV)).cpu().tolist() == logits.argmax(-1).tolist()[:1] + [77] + logits.argmax(-1).tolist()[2:]
    table = bf(100, 64, seed=4)
    toks = torch.tensor([3, 99, 0, 3])
    assert torch.equal(k.embed_gather(table.to(DEV), toks.to(DEV)).cpu(), table[toks])
    temp = torch.tensor([0.0, 1.0, 0.5]).to(DEV)
    u = torch.tensor([0.3, 0.0, 0.999999]).to(DEV)
    got = k.sample(logits.to(DEV), temp, u).cpu()
    assert got[0] == logits[0].argmax() and 0 <= got[1] < 4099 and 0 <= got[2] < 4099
    # inverse-CDF check for row 2
    p = torch.softmax(logits[2].double() / 0.5, -1).cumsum(0)
    assert abs(int(got[2]) - int((p > 0.999999).nonzero()[0])) <= 2 or p[int(got[2])] > 0.9999
    src = torch.arange(4 * 32, dtype=torch.float32).reshape(4, 32).to(DEV)
    dst = torch.zeros(6, 32, device=DEV)
    k.block_copy(dst, src, torch.tensor([5, 0]).to(DEV), torch.tensor([1, 3]).to(DEV))
    assert torch.equal(dst[5], src[1]) and torch.equal(dst[0], src[3]) and dst[1].sum() == 0


@pytest.mark.parametrize("M", [1, 2, 4, 8])
@pytest.mark.parametrize("N,Kd", [(520, 512), (2560, 1032), (37, 264), (6000, 256), (256, 4096), (1000, 2304)])
def test_gemv(M, N, Kd):
    k = K()
    W, x = bf(N, Kd, s=0.05, seed=5), bf(M, Kd, seed=6)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    k.gemv(W.to(DEV), x.to(DEV), out)
    close(out, x.float() @ W.float().t())
    out32 = torch.empty(M, N, dtype=torch.float32, device=DEV)
    k.gemv(W.to(DEV), x.to(DEV), out32)
    close(out32, x.float() @ W.float().t(), 1e-3)


@pytest.mark.parametrize("M,H,I", [(1, 520, 264), (4, 520, 264), (1, 4096, 256), (4, 2048, 520)])
def test_gemv_fused_norm_swiglu(M, H, I):
    """The last two shapes have few output rows and a long K: several CTAs share a 16-row block and
    the last one to arrive adds their partial sums (cross-CTA K split)."""
    k = K()
    Wgu, res, add = bf(2 * I, H, s=0.05, seed=7), bf(M, H, seed=8), bf(M, H, seed=9)
    gain = (1 + 0.1 * torch.randn(H)).float()
    out = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
    res_out = torch.empty(M, H, dtype=torch.bfloat16, device=DEV)
    k.gemv(Wgu.to(DEV), None, out, swiglu=True, norm=(res.to(DEV), add.to(DEV), gain.to(DEV), res_out, 1e-6))
    s, n = O.add_rms_norm(res, add, gain)
    n = n.to(torch.bfloat16).float()
    gu = n @ Wgu.float().t()
    close(res_out, s)
    close(out, O.silu_mul(gu[:, :I], gu[:, I:]), 3e-2)
    out2 = torch.empty(M, 2 * I, dtype=torch.bfloat16, device=DEV)
    k.gemv(Wgu.to(DEV), None, out2, norm=(res.to(DEV), None, gain.to(DEV), None, 1e-6))
    close(out2, O.rms_norm(res, gain).to(torch.bfloat16).float() @ Wgu.float().t())


@pytest.mark.parametrize("M,N,Kd,bn", [(128, 256, 64, 256), (200, 264, 192, 128), (300, 520, 1032, 0),
                                       (64, 64, 256, 64), (1000, 1536, 512, 256), (130, 136, 72, 128),
                                       (300, 520, 1032, 160), (2048, 2560, 1024, 0), (2048, 2560, 1024, 160),
                                       # CTA pairs (256-row tiles, 256 / 320 columns), edge tiles in both directions
                                       (300, 520, 1032, 1256), (300, 520, 1032, 1320), (257, 264, 72, 1320), (300, 520, 1032, 1288), (2048, 2560, 512, 1288),
                                       (1000, 1536, 512, 1256), (2048, 2560, 4096, 1320), (2100, 1288, 2560, 1256),
                                       # at most 128 rows: weights as the M operand, K in slices over a cluster
                                       (64, 2560, 4096, 0), (16, 12352, 2560, 0), (128, 520, 9216, 0), (5, 264, 520, 0)])
def test_gemm_tcgen05(M, N, Kd, bn):
    k = K()
    A, W = bf(M, Kd, seed=10), bf(N, Kd, s=0.05, seed=11)
    out = k.gemm(A.to(DEV), W.to(DEV), bn=bn)
    torch.cuda.synchronize()
    k.check_status()
    close(out, A.float() @ W.float().t())
    res = bf(M, N, seed=12)
    out = k.gemm(A.to(DEV), W.to(DEV), residual=res.to(DEV), bn=bn)
    torch.cuda.synchronize()
    k.check_status()
    close(out, A.float() @ W.float().t() + res.float())


@pytest.mark.parametrize("M,I,Kd", [(300, 128, 72), (1000, 776, 512), (2048, 9216, 2560), (257, 200, 1032), (64, 256, 128)])
def test_gemm_swiglu_epilogue(M, I, Kd):
    """Gate|up projection with silu(gate) * up taken in the CTA-pair GEMM's epilogue (64 rows: two-kernel fallback)."""
    k = K()
    A, W = bf(M, Kd, seed=20), bf(2 * I, Kd, s=0.05, seed=21)
    canary = torch.full((M + 1, I + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    out = k.gemm_swiglu(A.to(DEV), W.to(DEV), out=canary[:M, :I])
    torch.cuda.synchronize()
    k.check_status()
    gu = A.float() @ W.float().t()
    close(out, O.silu_mul(gu[:, :I], gu[:, I:]), 2e-2)
    assert bool((canary[M] == 7.0).all()) and bool((canary[:, I:] == 7.0).all()), "wrote outside the output"


@pytest.mark.parametrize("M,I,Kd", [(300, 128, 80), (1000, 776, 512), (2048, 2176, 1024)])
def test_gemm_i8_swiglu_epilogue(M, I, Kd):
    k = K()
    g = torch.Generator().manual_seed(9)
    Aq = torch.randint(-127, 128, (M, Kd), generator=g, dtype=torch.int8)
    Wq = torch.randint(-127, 128, (2 * I, Kd), generator=g, dtype=torch.int8)
    sa, sw = torch.rand(M, generator=g) * 0.01 + 1e-3, torch.rand(2 * I, generator=g) * 0.002 + 1e-4
    out = k.gemm_i8_swiglu(Aq.to(DEV), sa.to(DEV), Wq.to(DEV), sw.to(DEV))
    torch.cuda.synchronize()
    k.check_status()
    gu = ((Aq.double() @ Wq.double().t()) * sa.double()[:, None] * sw.double()[None, :]).float()
    close(out, O.silu_mul(gu[:, :I], gu[:, I:]), 1e-2)


@pytest.mark.parametrize("M,N,Kd,bn", [(128, 256, 128, 256), (200, 264, 400, 128), (77, 520, 1040, 0),
                                       (300, 488, 528, 160), (64, 2560, 4096, 0), (16, 520, 9216, 0),
                                       # CTA pairs
                                       (300, 488, 528, 1256), (300, 488, 528, 1320), (300, 488, 528, 1288), (1000, 1536, 512, 0),
                                       (2048, 2560, 4096, 1320)])
def test_gemm_i8_tcgen05(M, N, Kd, bn):
    k = K()
    g = torch.Generator().manual_seed(13)
    Aq = torch.randint(-127, 128, (M, Kd), generator=g, dtype=torch.int8)
    Wq = torch.randint(-127, 128, (N, Kd), generator=g, dtype=torch.int8)
    sa, sw = torch.rand(M, generator=g) * 0.01 + 1e-3, torch.rand(N, generator=g) * 0.01 + 1e-3
    out = k.gemm_i8(Aq.to(DEV), sa.to(DEV), Wq.to(DEV), sw.to(DEV), bn=bn)
    torch.cuda.synchronize()
    k.check_status()
    ref = (Aq.double() @ Wq.double().t()) * sa.double()[:, None] * sw.double()[None, :]
    close(out, ref.float(), 1e-2)


def _gdn_inputs(T, nk, nv, dk, dv, seed):
    conv_dim = 2 * nk * dk + nv * dv
    ldp = (conv_dim + nv * dv + 2 * nv + 7) // 8 * 8     # rows are 16-byte aligned, as in the model
    proj = bf(T, ldp, seed=seed)
    g = torch.Generator().manual_seed(seed + 100)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.3).float()
    A_log = torch.log(1 + 15 * torch.rand(nv, generator=g))
    dt_bias = torch.randn(nv, generator=g) * 0.5
    norm_w = 1 + 0.1 * torch.randn(dv, generator=g)
    return proj, conv_w, A_log, dt_bias, norm_w, conv_dim


def _gdn_oracle(proj, conv_w, A_log, dt_bias, norm_w, nk, nv, dk, dv, conv_state, state):
    """fp32 oracle over T rows: returns the normed outputs, updates states in place."""
    T = proj.shape[0]
    conv_dim = 2 * nk * dk + nv * dv
    p = proj.float()
    qkv, z = p[:, :conv_dim], p[:, conv_dim:conv_dim + nv * dv]
    b, a = p[:, conv_dim + nv * dv:conv_dim + nv * dv + nv], p[:, conv_dim + nv * dv + nv:conv_dim + nv * dv + 2 * nv]
    conv, new_conv = O.conv1d_silu_seq(conv_w, qkv, conv_state)
    conv_state.copy_(new_conv)
    q = conv[:, :nk * dk].reshape(T, nk, dk)
    kk = conv[:, nk * dk:2 * nk * dk].reshape(T, nk, dk)
    v = conv[:, 2 * nk * dk:].reshape(T, nv, dv)
    qn, kn, beta, g = O.gdn_head_prep(q, kk, b, a, A_log, dt_bias, nv // nk)
    o = O.delta_recurrent(qn, kn, v, beta, g, state)
    return O.rms_norm_gated(o, norm_w, z.reshape(T, nv, dv)).reshape(T, nv * dv)


@pytest.mark.parametrize("nk,nv,dk,dv", [(2, 4, 64, 64), (2, 4, 128, 128), (2, 6, 128, 128)])
def test_gdn_decode_steps_and_verify(nk, nv, dk, dv):
    k = K()
    T = 9
    proj, conv_w, A_log, dt_bias, norm_w, conv_dim = _gdn_inputs(T, nk, nv, dk, dv, 20)
    conv_state, state = torch.zeros(conv_dim, 3), torch.zeros(nv, dk, dv)
    ref = _gdn_oracle(proj, conv_w, A_log, dt_bias, norm_w, nk, nv, dk, dv, conv_state, state)
    d = lambda t: t.to(DEV)
    ring = torch.zeros(3, k.RING, conv_dim, dtype=torch.bfloat16, device=DEV)
    st = torch.zeros(3, nv, dk, dv, device=DEV)
    slots = torch.tensor([2], dtype=torch.int32, device=DEV)
    out = torch.empty(T, nv * dv, dtype=torch.bfloat16, device=DEV)
    cw, al, db, nw = d(conv_w), d(A_log), d(dt_bias), d(norm_w.float())
    for t in range(5):      # five single-token steps
        pos = torch.tensor([t], dtype=torch.int32, device=DEV)
        k.gdn_decode(d(proj[t:t + 1]), cw, al, db, nw, ring, st, slots, pos, out[t:t + 1], nk=nk, nv=nv, dk=dk,
                     dv=dv, eps=1e-6)
    # then a 4-token verify chain that leaves the state untouched and records the updates
    rec = torch.zeros(1, 4, nv, dk + dv + 1, device=DEV)
    base = st.clone()
    pos = torch.tensor([5], dtype=torch.int32, device=DEV)
    k.gdn_decode(d(proj[5:9]), cw, al, db, nw, ring, st, slots, pos, out[5:9], nk=nk, nv=nv, dk=dk, dv=dv,
                 eps=1e-6, ntok=4, record=rec, write_state=False)
    assert torch.equal(st, base)
    close(out, ref, 3e-2)
    k.gdn_commit(st, rec, slots, torch.tensor([4], dtype=torch.int32, device=DEV), nv=nv, dk=dk, dv=dv)
    close(st[2], state, 1e-3)
    assert st[0].abs().sum() == 0


@pytest.mark.parametrize("mode", [3, 2, 1])
@pytest.mark.parametrize("nk,nv,dk,dv,T1,T2", [(2, 4, 64, 64, 150, 37), (2, 4, 128, 128, 64, 70), (1, 2, 128, 128, 5, 3),
                                               (2, 4, 128, 128, 700, 333)])
def test_gdn_prefill_chunked(nk, nv, dk, dv, T1, T2, mode):
    """mode 3: prep fused into the TF32 prepare kernel + bf16-operand scan (three-stage operand ring); mode 2: the
    same with the prep kernel as its own launch; mode 1: TF32 for both."""
    k = K()
    k.call("set_gdn_tc", mode)
    try:
        _gdn_prefill_case(k, nk, nv, dk, dv, T1, T2, mode)
    finally:
        k.call("set_gdn_tc", 3)


def _gdn_prefill_case(k, nk, nv, dk, dv, T1, T2, mode):
    T = T1 + T2
    proj, conv_w, A_log, dt_bias, norm_w, conv_dim = _gdn_inputs(T, nk, nv, dk, dv, 30)
    conv_state, state = torch.zeros(conv_dim, 3), torch.zeros(nv, dk, dv)
    ref = _gdn_oracle(proj, conv_w, A_log, dt_bias, norm_w, nk, nv, dk, dv, conv_state, state)
    d = lambda t: t.to(DEV)
    ring = torch.zeros(k.RING, conv_dim, dtype=torch.bfloat16, device=DEV)
    st = torch.zeros(nv, dk, dv, device=DEV)
    out = torch.empty(T, nv * dv, dtype=torch.bfloat16, device=DEV)
    scratch = torch.empty(k.gdn_prefill_scratch_floats(max(T1, T2), nk, nv, dk, dv), device=DEV)
    args = (d(conv_w), d(A_log), d(dt_bias), d(norm_w.float()), ring, st, scratch)
    pj = d(proj)
    k.gdn_prefill(pj[:T1], *args, out[:T1], pos0=0, nk=nk, nv=nv, dk=dk, dv=dv, eps=1e-6)
    k.gdn_prefill(pj[T1:], *args, out[T1:], pos0=T1, nk=nk, nv=nv, dk=dk, dv=dv, eps=1e-6)
    close(out, ref, 3e-2)
    # the chunk products run as TF32 (10-bit mantissa) or, in the scan of mode 2, with bf16 operands
    close(st, state, 4e-3 if mode == 1 else 2e-2)
    # a decode step after the chunked prefill continues from the ring + state
    extra = bf(1, proj.shape[1], seed=31)
    ref2 = _gdn_oracle(extra, conv_w, A_log, dt_bias, norm_w, nk, nv, dk, dv, conv_state, state)
    out2 = torch.empty(1, nv * dv, dtype=torch.bfloat16, device=DEV)
    k.gdn_decode(d(extra), d(conv_w), d(A_log), d(dt_bias), d(norm_w.float()), ring.unsqueeze(0), st.unsqueeze(0),
                 torch.zeros(1, dtype=torch.int32, device=DEV), torch.tensor([T], dtype=torch.int32, device=DEV),
                 out2, nk=nk, nv=nv, dk=dk, dv=dv, eps=1e-6)
    close(out2, ref2, 3e-2)


def _attn_setup(T, nh, nkv, hd, rot, seed):
    ldp = nh * 2 * hd + 2 * nkv * hd
    proj = bf(T, ldp, seed=seed)
    g = torch.Generator().manual_seed(seed + 1)
    qg, kg = 1 + 0.1 * torch.randn(hd, generator=g), 1 + 0.1 * torch.randn(hd, generator=g)
    cos, sin = O.rope_tables(rot, 1e7, 4096)
    return proj, qg.float(), kg.float(), cos, sin


def _attn_oracle(proj, qg, kg, cos, sin, nh, nkv, hd, rot, pos):
    T = proj.shape[0]
    p = proj.float()
    qgate = p[:, :nh * 2 * hd].reshape(T, nh, 2 * hd)
    q, gate = qgate[..., :hd], qgate[..., hd:]
    kk = p[:, nh * 2 * hd:nh * 2 * hd + nkv * hd].reshape(T, nkv, hd)
    v = p[:, nh * 2 * hd + nkv * hd:].reshape(T, nkv, hd)
    q = O.apply_rope(O.rms_norm(q, qg), cos[pos], sin[pos], rot)
    kk = O.apply_rope(O.rms_norm(kk, kg), cos[pos], sin[pos], rot)
    return O.gated_attention(q, gate, kk, v, pos, hd ** -0.5).reshape(T, nh * hd), kk, v


@pytest.mark.parametrize("nh,nkv,hd,rot,T1,T2", [(4, 2, 64, 16, 100, 30), (4, 1, 256, 64, 70, 129), (2, 2, 256, 64, 3, 1)])
def test_attention_prefill_and_decode(nh, nkv, hd, rot, T1, T2):
    k = K()
    T = T1 + T2 + 3
    proj, qg, kg, cos, sin = _attn_setup(T, nh, nkv, hd, rot, 40)
    pos = torch.arange(T)
    ref, kref, vref = _attn_oracle(proj, qg, kg, cos, sin, nh, nkv, hd, rot, pos)
    d = lambda t: t.to(DEV)
    nblk = (T + 63) // 64
    pool_blocks = nblk + 3
    kpool = torch.zeros(pool_blocks * 64, nkv, hd, dtype=torch.bfloat16, device=DEV)
    vpool = torch.zeros_like(kpool)
    bt = torch.tensor(list(range(pool_blocks - 1, pool_blocks - 1 - nblk, -1)), dtype=torch.int32)  # reversed blocks
    slot_of = lambda p: int(bt[p // 64]) * 64 + p % 64
    out = torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV)
    pj, dc, ds = d(proj), d(cos), d(sin)
    for s, e in ((0, T1), (T1, T1 + T2)):
        n = e - s
        q = torch.empty(n, nh, hd, dtype=torch.bfloat16, device=DEV)
        slots = torch.tensor([slot_of(p) for p in range(s, e)], dtype=torch.int32, device=DEV)
        ridx = torch.arange(s, e, dtype=torch.int32, device=DEV)
        k.attn_prep(pj[s:e], d(qg), d(kg), dc, ds, ridx, slots, q, kpool, vpool, nh=nh, nkv=nkv, hd=hd, rot=rot, eps=1e-6)
        k.attn_prefill(q, pj[s:e], kpool, vpool, d(bt), out[s:e], q_pos0=s, nh=nh, nkv=nkv, hd=hd)
    # three decode steps (2 rows in the bucket: row 1 is padding)
    nsplit = 3
    part_o = torch.empty(2, nh, nsplit, hd, device=DEV)
    part_ml = torch.empty(2, nh, nsplit, 2, device=DEV)
    tickets = torch.zeros(2, nkv, dtype=torch.int32, device=DEV)
    btab = torch.zeros(2, nblk, dtype=torch.int32)
    btab[0] = bt
    for p in range(T1 + T2, T):
        posv = torch.tensor([p, -1], dtype=torch.int32, device=DEV)
        o2 = torch.empty(2, nh * hd, dtype=torch.bfloat16, device=DEV)
        pr = torch.cat([pj[p:p + 1], pj[p:p + 1]])
        k.attn_decode(pr, d(qg), d(kg), dc, ds, posv, posv.clamp_min(0), d(btab), kpool, vpool, part_o, part_ml, tickets, o2,
                      nh=nh, nkv=nkv, hd=hd, rot=rot, nsplit=nsplit, eps=1e-6)
        out[p] = o2[0]
    close(out, ref, 3e-2)
    got_k = torch.stack([kpool[slot_of(p)] for p in range(T)]).cpu()
    close(got_k, kref, 2e-2)


@pytest.mark.parametrize("nh,nkv,hd,rot,chunks", [(4, 2, 64, 16, (200, 57, 300)), (4, 1, 256, 64, (130, 128, 333)),
                                                  (2, 2, 256, 64, (64, 1000))])
def test_attention_prefill_tcgen05_matches_oracle_and_the_mma_kernel(nh, nkv, hd, rot, chunks):
    """Chunked causal prefill through the tcgen05 kernel (TMA pages, TMEM accumulators, lazy rescale)
    against the fp32 oracle and the mma.sync kernel: chunk starts that are not page aligned, query
    tiles with padded rows, scattered pages, the output gate; run twice for bit-equal results."""
    k = K()
    T = sum(chunks)
    proj, qg, kg, cos, sin = _attn_setup(T, nh, nkv, hd, rot, 41)
    qg = qg * 6.0                                  # scores ~ N(0, 6^2): the running maximum moves by more than 2^8, rescales happen
    pos = torch.arange(T)
    ref, _, _ = _attn_oracle(proj, qg, kg, cos, sin, nh, nkv, hd, rot, pos)
    d = lambda t: t.to(DEV)
    nblk = (T + 63) // 64
    kpool = torch.zeros((nblk + 2) * 64, nkv, hd, dtype=torch.bfloat16, device=DEV)
    vpool = torch.zeros_like(kpool)
    perm = torch.randperm(nblk + 1, generator=torch.Generator().manual_seed(3))[:nblk] + 1
    bt = perm.to(torch.int32)
    pj, dc, ds = d(proj), d(cos), d(sin)
    outs = {}
    for tc in (True, False, True):
        k.ATTN_TC = tc
        out = torch.full((T + 1, nh * hd), 7.0, dtype=torch.bfloat16, device=DEV)      # last row: canary
        s = 0
        try:
            for n in chunks:
                e = s + n
                q = torch.empty(n, nh, hd, dtype=torch.bfloat16, device=DEV)
                slots = (bt.long()[torch.arange(s, e) // 64] * 64 + torch.arange(s, e) % 64).to(torch.int32).to(DEV)
                ridx = torch.arange(s, e, dtype=torch.int32, device=DEV)
                k.attn_prep(pj[s:e], d(qg), d(kg), dc, ds, ridx, slots, q, kpool, vpool, nh=nh, nkv=nkv, hd=hd, rot=rot, eps=1e-6)
                k.attn_prefill(q, pj[s:e], kpool, vpool, d(bt), out[s:e], q_pos0=s, nh=nh, nkv=nkv, hd=hd)
                s = e
        finally:
            k.ATTN_TC = True
        torch.cuda.synchronize()
        k.check_status()
        assert bool((out[T] == 7.0).all()), "wrote past the last row"
        outs.setdefault(tc, []).append(out[:T].clone())
    close(outs[True][0], ref, 3e-2)
    close(outs[False][0], ref, 3e-2)
    assert torch.equal(outs[True][0], outs[True][1]), "the tcgen05 kernel must be deterministic"
    # per element against the mma.sync kernel (both round P to bf16; accumulation order differs)
    a, b = outs[True][0].float(), outs[False][0].float()
    assert float((a - b).abs().max()) <= 0.03 * float(b.abs().max())


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("N,Kd", [(520, 512), (2560, 1040), (37, 272)])
def test_gemv_i8_w8a8(M, N, Kd):
    k = K()
    from coffin_b200.weights.quant import QWeight
    W, x = bf(N, Kd, s=0.05, seed=50), bf(M, Kd, seed=51)
    q = QWeight.quantize(W.float())
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    k.gemv_i8(q.wq.to(DEV), q.scale.to(DEV), x.to(DEV), out)
    close(out, O.w8a8_linear(x, q.wq, q.scale), 5e-3)
    # fused norm + swiglu
    I = N // 2
    res, add = bf(M, Kd, seed=52), bf(M, Kd, seed=53)
    gain = (1 + 0.1 * torch.randn(Kd)).float()
    out2 = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
    ro = torch.empty(M, Kd, dtype=torch.bfloat16, device=DEV)
    k.gemv_i8(q.wq[:2 * I].to(DEV), q.scale[:2 * I].to(DEV), None, out2, swiglu=True,
              norm=(res.to(DEV), add.to(DEV), gain.to(DEV), ro, 1e-6))
    s_, n_ = O.add_rms_norm(res, add, gain)
    gu = O.w8a8_linear(n_.to(torch.bfloat16), q.wq[:2 * I], q.scale[:2 * I])
    close(ro, s_)
    close(out2, O.silu_mul(gu[:, :I], gu[:, I:]), 3e-2)


def test_quant_rows_and_i8_prefill_chain():
    k = K()
    from coffin_b200.weights.quant import QWeight
    x = bf(70, 528, seed=60)
    qx, sx = k.quant_rows(x.to(DEV))
    rq, rs = O.quant_rows_int8(x, floor=1e-8)
    assert (qx.cpu().int() - rq.int()).abs().max() <= 1 and torch.allclose(sx.cpu(), rs, rtol=1e-5)
    W = bf(264, 528, s=0.05, seed=61)
    q = QWeight.quantize(W.float())
    out = k.gemm_i8(qx, sx, q.wq.to(DEV), q.scale.to(DEV))
    torch.cuda.synchronize()
    k.check_status()
    close(out, O.w8a8_linear(x, q.wq, q.scale), 1e-2)
    gu = bf(9, 2 * 264, seed=62)
    qs, ss = k.quant_rows(gu.to(DEV), swiglu=True)
    ref = O.silu_mul(gu[:, :264], gu[:, 264:]).to(torch.bfloat16)
    rq2, rs2 = O.quant_rows_int8(ref, floor=1e-8)
    assert (qs.cpu().int() - rq2.int()).abs().max() <= 1
    # the norm kernel's own int8 output: bit-equal to quantising its bf16 output, with and without the add
    xr, add = bf(33, 528, seed=63).to(DEV), bf(33, 528, seed=64).to(DEV)
    gain = (1 + 0.1 * torch.randn(528)).float().to(DEV)
    for a in (None, add):
        normed = k.rmsnorm(xr, gain, 1e-6, add=a, res_out=torch.empty_like(xr) if a is not None else None)
        q_ref, s_ref = k.quant_rows(normed)
        q8 = torch.empty(33, 528, dtype=torch.int8, device=DEV)
        s8 = torch.empty(33, dtype=torch.float32, device=DEV)
        ro = torch.empty_like(xr) if a is not None else None
        k.rmsnorm(xr, gain, 1e-6, add=a, res_out=ro, quant=(q8, s8))
        assert torch.equal(q8, q_ref) and torch.equal(s8, s_ref)


@pytest.mark.parametrize("M,N,Kd", [(1, 520, 512), (4, 2560, 1024), (8, 264, 256), (2, 1000, 2304)])
def test_gemv_w4a8(M, N, Kd):
    """W4A8 GEMV against the integer oracle (group-128 int4 weights, per-token int8 activations)."""
    k = K()
    from coffin_b200.weights.quant import W4A8Weight
    W, x = bf(N, Kd, s=0.05, seed=60), bf(M, Kd, seed=61)
    q = W4A8Weight.quantize(W.float())
    wq, sc = q.to_nk()
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    k.gemv_w4(wq.to(DEV), sc.to(DEV), x.to(DEV), out)
    close(out, O.w4a8_linear(x, q.packed, q.scale, Kd), 5e-3)
    close(k.w4_dequant(wq.to(DEV), sc.to(DEV)), q.dequant(), 1e-2)
    # fused norm + swiglu
    I = N // 2 // 8 * 8
    res, add = bf(M, Kd, seed=62), bf(M, Kd, seed=63)
    gain = (1 + 0.1 * torch.randn(Kd)).float()
    out2 = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
    ro = torch.empty(M, Kd, dtype=torch.bfloat16, device=DEV)
    q2 = W4A8Weight.quantize(W[:2 * I].float())
    wq2, sc2 = q2.to_nk()
    k.gemv_w4(wq2.to(DEV), sc2.to(DEV), None, out2, swiglu=True, norm=(res.to(DEV), add.to(DEV), gain.to(DEV), ro, 1e-6))
    s_, n_ = O.add_rms_norm(res, add, gain)
    gu = O.w4a8_linear(n_.to(torch.bfloat16), q2.packed, q2.scale, Kd)
    close(ro, s_)
    close(out2, O.silu_mul(gu[:, :I], gu[:, I:]), 3e-2)


def test_moe_gemv_w4a8_slots():
    k = K()
    from coffin_b200.weights.quant import W4A8Weight
    E, I, H = 6, 128, 256
    g = torch.Generator().manual_seed(70)
    Wgu = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(3, H, generator=g).to(torch.bfloat16)
    q = W4A8Weight.quantize(Wgu.float())
    wq, sc = q.to_nk()
    slot_e = torch.tensor([4, 0, -1, 5, 1], dtype=torch.int32, device=DEV)
    slot_x = torch.tensor([0, 0, 1, 2, 2], dtype=torch.int32, device=DEV)
    out = torch.zeros(5, I, dtype=torch.bfloat16, device=DEV)
    k.moe_gemv_w4(wq.to(DEV), sc.to(DEV), x.to(DEV), out, slot_e, slot_x, swiglu=True)
    for s in range(5):
        e, r = int(slot_e[s]), int(slot_x[s])
        if e < 0:
            assert float(out[s].abs().max()) == 0.0
            continue
        gu = O.w4a8_linear(x[r:r + 1], q.packed[e], q.scale[e], H)
        close(out[s:s + 1], O.silu_mul(gu[:, :I], gu[:, I:]), 3e-2)


def test_moe_gemv_i8_slots():
    """Routed experts from int8 stacks, one slot per (expert, activation row): the kernel quantises the row
    itself; against the dequantised weights times the quantised row in fp32."""
    k = K()
    from coffin_b200.weights.quant import QWeight
    E, I, H = 6, 128, 256
    g = torch.Generator().manual_seed(71)
    q = QWeight.quantize(torch.randn(E, 2 * I, H, generator=g) * 0.05)
    qd = QWeight.quantize(torch.randn(E, H, I, generator=g) * 0.05)
    x = torch.randn(3, H, generator=g).to(torch.bfloat16)
    slot_e = torch.tensor([4, 0, -1, 5, 1], dtype=torch.int32, device=DEV)
    slot_x = torch.tensor([0, 0, 1, 2, 2], dtype=torch.int32, device=DEV)
    out = torch.zeros(5, I, dtype=torch.bfloat16, device=DEV)
    k.moe_gemv_i8(q.wq.to(DEV), q.scale.to(DEV), x.to(DEV), out, slot_e, slot_x, swiglu=True)
    y = torch.zeros(5, H, dtype=torch.float32, device=DEV)
    k.moe_gemv_i8(qd.wq.to(DEV), qd.scale.to(DEV), out, y, slot_e, None)

    def qrow(v):                                   # the per-row activation quantisation of the kernel
        sc = v.float().abs().amax().clamp_min(1e-8) / 127.0
        return (v.float() / sc).round().clamp(-127, 127) * sc

    for s in range(5):
        e, r = int(slot_e[s]), int(slot_x[s])
        if e < 0:
            assert float(out[s].abs().max()) == 0.0 and float(y[s].abs().max()) == 0.0
            continue
        gu = qrow(x[r]) @ q.dequant()[e].T
        close(out[s:s + 1], O.silu_mul(gu[None, :I], gu[None, I:]), 2e-2)
        close(y[s:s + 1], (qrow(out[s].cpu()) @ qd.dequant()[e].T)[None], 2e-2)


@pytest.mark.parametrize("T,k,E,H,N", [(300, 4, 8, 256, 512), (64, 2, 16, 128, 264), (1000, 8, 32, 512, 256), (513, 2, 4, 2048, 160)])
def test_grouped_gemm_from_int8_stacks(T, k, E, H, N):
    """Grouped kind::i8 tcgen05 GEMM over expert-sorted int8 rows: per-row activation scales times the
    expert's per-column weight scales in the epilogue; against the dequantised fp32 product per expert.
    Slots of no local expert (-1) are left out; rows behind the tile list stay untouched (canary)."""
    from coffin_b200.weights.quant import QWeight
    kk = K()
    g = torch.Generator().manual_seed(T + E + 1)
    idx = torch.randint(-2, E, (T, k), generator=g, dtype=torch.int32)
    x = (torch.randn(T, H, generator=g) * 0.5).bfloat16()
    qw = QWeight.quantize(torch.randn(E, N, H, generator=g) * 0.05)
    d = kk.moe_dispatch(idx.to(DEV), E)
    pos = d["pos"].cpu().reshape(T, k)
    xq, xs = kk.quant_rows(x.to(DEV))
    out = torch.full((T * k, N), 7.0, dtype=torch.bfloat16, device=DEV)
    y = kk.gemm_i8_grouped(xq.index_select(0, d["src_tok"]), xs.index_select(0, d["src_tok"]), qw.wq.to(DEV),
                           qw.scale.to(DEV), d, out=out).float().cpu()
    kk.check_status()
    xdq = xq.float().cpu() * xs.cpu()[:, None]
    Wd = qw.dequant()
    for t in range(0, T, 5):
        for j in range(k):
            e = int(idx[t, j])
            if e < 0:
                continue
            ref = xdq[t] @ Wd[e].T
            got = y[pos[t, j]]
            assert (got - ref).abs().max() <= 1e-2 * ref.abs().max() + 1e-3
    n_local = int((idx >= 0).sum())
    assert bool((y[n_local:] == 7.0).all())
    y2 = kk.gemm_i8_grouped(xq.index_select(0, d["src_tok"]), xs.index_select(0, d["src_tok"]), qw.wq.to(DEV),
                            qw.scale.to(DEV), d).float().cpu()
    assert torch.equal(y2[:n_local], y[:n_local])


@pytest.mark.parametrize("T,k,E,H,N", [(300, 4, 8, 256, 512), (64, 2, 16, 128, 264), (1000, 8, 32, 512, 256)])
def test_moe_dispatch_and_grouped_gemm(T, k, E, H, N):
    """Device-side expert-major dispatch + grouped tcgen05 GEMM against a per-expert fp32 matmul;
    some slots belong to no local expert (-1) and must be left out."""
    kk = K()
    g = torch.Generator().manual_seed(T + E)
    idx = torch.randint(-2, E, (T, k), generator=g, dtype=torch.int32)
    x = (torch.randn(T, H, generator=g) * 0.5).bfloat16()
    W = (torch.randn(E, N, H, generator=g) * 0.05).bfloat16()
    d = kk.moe_dispatch(idx.to(DEV), E)
    pos = d["pos"].cpu().reshape(T, k)
    src = d["src_tok"].cpu()
    n_local = int((idx >= 0).sum())
    assert sorted(pos[idx >= 0].tolist()) == list(range(n_local))
    assert (pos[idx < 0] == -1).all()
    nt = int(d["count"].cpu())
    row0, rows, ex = d["row0"].cpu()[:nt], d["rows"].cpu()[:nt], d["expert"].cpu()[:nt]
    assert int(rows.sum()) == n_local and int(rows.max()) <= 128
    for t in range(T):
        for j in range(k):
            if idx[t, j] >= 0:
                assert src[pos[t, j]] == t
    xs = x.to(DEV).index_select(0, d["src_tok"])
    y = kk.gemm_grouped(xs, W.to(DEV), d).float().cpu()
    for t in range(0, T, 7):
        for j in range(k):
            e = int(idx[t, j])
            if e < 0:
                continue
            ref = x[t].float() @ W[e].float().T
            got = y[pos[t, j]]
            assert (got - ref).abs().max() <= 2e-2 * ref.abs().max() + 1e-3
    # every tile stays inside one expert's row range
    for i in range(nt):
        sel = (pos >= int(row0[i])) & (pos < int(row0[i] + rows[i]))
        assert (idx[sel] == int(ex[i])).all()


@pytest.mark.parametrize("T,k,E,H,I", [(300, 4, 8, 512, 256), (700, 8, 32, 1024, 512), (64, 2, 16, 512, 264), (2048, 8, 64, 2048, 512)])
def test_grouped_gemm_from_int4_codes(T, k, E, H, I):
    """Routed-expert prefill from the int4 stacks: codes expanded inside the CTA, gate|up with the SwiGLU
    epilogue, then the down projection; against the dequantised fp32 product per expert."""
    from coffin_b200.weights.quant import W4A8Weight
    kk = K()
    g = torch.Generator().manual_seed(T + E)
    idx = torch.randint(-1, E, (T, k), generator=g, dtype=torch.int32)
    x = (torch.randn(T, H, generator=g) * 0.5).bfloat16()
    qgu = W4A8Weight.quantize(torch.randn(E, 2 * I, H, generator=g) * 0.05)
    down = I % 512 == 0                  # the kernel takes reduction lengths that are multiples of 512
    Wgu = qgu.dequant().float()          # [E, 2I, H]
    if down:
        qdn = W4A8Weight.quantize(torch.randn(E, H, I, generator=g) * 0.05)
        Wdn = qdn.dequant().float()      # [E, H, I]
    d = kk.moe_dispatch(idx.to(DEV), E)
    pos = d["pos"].cpu().reshape(T, k)
    xs = x.to(DEV).index_select(0, d["src_tok"])
    gq, gs = (t.to(DEV) for t in qgu.to_nk())
    inter = kk.gemm_w4_grouped(xs, gq, gs, d, swiglu=True)
    if down:
        dq, ds = (t.to(DEV) for t in qdn.to_nk())
        y = kk.gemm_w4_grouped(inter, dq, ds, d)
    torch.cuda.synchronize()
    kk.check_status()
    # plain (no SwiGLU) form of the first projection as well
    gu_plain = kk.gemm_w4_grouped(xs, gq, gs, d)
    torch.cuda.synchronize()
    kk.check_status()
    inter_c, gu_c = inter.float().cpu(), gu_plain.float().cpu()
    y_c = y.float().cpu() if down else None
    for t in range(0, T, 5):
        for j in range(k):
            e = int(idx[t, j])
            if e < 0:
                continue
            gu = x[t].float() @ Wgu[e].T
            ref_i = O.silu_mul(gu[None, :I], gu[None, I:])[0]
            got_i = inter_c[pos[t, j]]
            assert (got_i - ref_i).abs().max() <= 2e-2 * ref_i.abs().max() + 1e-3, f"inter t={t} j={j}"
            assert (gu_c[pos[t, j]] - gu).abs().max() <= 2e-2 * gu.abs().max() + 1e-3, f"gate|up t={t} j={j}"
            if down:
                ref_y = got_i.bfloat16().float() @ Wdn[e].T
                assert (y_c[pos[t, j]] - ref_y).abs().max() <= 2e-2 * ref_y.abs().max() + 1e-3, f"down t={t} j={j}"


@pytest.mark.parametrize("nh,nkv,T1", [(16, 4, 150), (8, 4, 64), (6, 2, 257)])
def test_attention_decode_batch_kernel(nh, nkv, T1):
    """Tensor-core batch decode kernel (one CTA per row and kv head) against the fp32 oracle and the
    split kernel: every row has its own blocks holding the same prefix, one row is padding."""
    from coffin_b200.ops import _lib
    k = K()
    hd, rot, R = 256, 64, 33
    T = T1 + 1
    proj, qg, kg, cos, sin = _attn_setup(T, nh, nkv, hd, rot, 77)
    ref, _, _ = _attn_oracle(proj, qg, kg, cos, sin, nh, nkv, hd, rot, torch.arange(T))
    d = lambda t: t.to(DEV)
    nblk = (T + 63) // 64
    kpool = torch.zeros((R * nblk + 1) * 64, nkv, hd, dtype=torch.bfloat16, device=DEV)
    vpool = torch.zeros_like(kpool)
    pj, dc, ds = d(proj), d(cos), d(sin)
    btab = torch.zeros(R, nblk, dtype=torch.int32)
    for r in range(R):
        btab[r] = torch.arange(1 + r * nblk, 1 + (r + 1) * nblk)
    # prefix K/V through the prep kernel into row 0's blocks, then copied to every other row's blocks
    q = torch.empty(T1, nh, hd, dtype=torch.bfloat16, device=DEV)
    slots = torch.tensor([int(btab[0, p // 64]) * 64 + p % 64 for p in range(T1)], dtype=torch.int32, device=DEV)
    k.attn_prep(pj[:T1], d(qg), d(kg), dc, ds, torch.arange(T1, dtype=torch.int32, device=DEV), slots, q, kpool, vpool,
                nh=nh, nkv=nkv, hd=hd, rot=rot, eps=1e-6)
    for r in range(1, R):
        for b in range(nblk):
            s0, s1 = int(btab[0, b]) * 64, int(btab[r, b]) * 64
            kpool[s1:s1 + 64] = kpool[s0:s0 + 64]
            vpool[s1:s1 + 64] = vpool[s0:s0 + 64]
    posv = torch.full((R,), T1, dtype=torch.int32)
    posv[5] = -1
    posv = posv.to(DEV)
    pr = pj[T1:T1 + 1].repeat(R, 1).contiguous()
    nsplit = 2
    outs = []
    for thr in (1, 0):               # 1: batch kernel for any size; 0: split kernel
        _lib.call_nostream("set_attn_batch_ctas", thr)
        kp, vp = kpool.clone(), vpool.clone()
        part_o = torch.empty(R, nh, nsplit, hd, device=DEV)
        part_ml = torch.empty(R, nh, nsplit, 2, device=DEV)
        tickets = torch.zeros(R, nkv, dtype=torch.int32, device=DEV)
        o2 = torch.zeros(R, nh * hd, dtype=torch.bfloat16, device=DEV)
        k.attn_decode(pr, d(qg), d(kg), dc, ds, posv, posv.clamp_min(0), d(btab), kp, vp, part_o, part_ml, tickets, o2,
                      nh=nh, nkv=nkv, hd=hd, rot=rot, nsplit=nsplit, eps=1e-6)
        outs.append(o2.float().cpu())
        # the appended key landed in every live row's block
        for r in (0, R - 1):
            slot = int(btab[r, T1 // 64]) * 64 + T1 % 64
            assert kp[slot].float().abs().sum() > 0
    _lib.call_nostream("set_attn_batch_ctas", 32)
    for r in range(R):
        if r == 5:
            continue
        close(outs[0][r], ref[T1], 3e-2)
        close(outs[0][r], outs[1][r], 2e-2)


CANARY = -12345.0


def _guarded(rows, cols, dtype):
    """An output tensor carved out of a larger buffer whose margins hold a canary value."""
    pad = 64
    buf = torch.full((rows + 2, cols + 2 * pad), CANARY, dtype=dtype, device=DEV)
    return buf, buf[1:1 + rows, pad:pad + cols]


def _intact(buf, rows, cols):
    pad = 64
    ok = bool((buf[0] == CANARY).all()) and bool((buf[-1] == CANARY).all())
    return ok and bool((buf[1:1 + rows, :pad] == CANARY).all()) and bool((buf[1:1 + rows, pad + cols:] == CANARY).all())


@pytest.mark.parametrize("M,N,Kd", [(1, 2560, 9216), (8, 2560, 4096), (4, 1000, 520), (40, 2560, 4096), (64, 520, 1024)])
def test_projections_stay_in_bounds_and_repeat_bit_exact(M, N, Kd):
    """Kernels that split K over CTAs (the tensor-core GEMV for narrow outputs, which finishes through arrival
    tickets; the tcgen05 product of few rows, which adds its slices over a cluster): outputs written into a canary-padded
    buffer leave the canaries alone, and a second run of the same launch gives the same bits (partial
    sums are added in slice order, never in arrival order)."""
    k = K()
    x, W = bf(M, Kd, seed=1).to(DEV), bf(N, Kd, s=0.05, seed=2).to(DEV)
    ref = x.float().cpu() @ W.float().cpu().t()
    runs = []
    for _ in range(2):
        buf, out = _guarded(M, N, torch.bfloat16)
        if M <= 8:
            k.gemv(W, x, out)
        else:
            k.gemm(x, W, out=out)
        torch.cuda.synchronize()
        assert _intact(buf, M, N)
        runs.append(out.clone())
    assert torch.equal(runs[0], runs[1])
    close(runs[0], ref)
    k.check_status()


def test_argmax_and_attention_tickets_repeat_bit_exact():
    """The ticketed reductions (two-stage arg-max, split-KV merge by the last split to arrive) re-arm
    themselves: back-to-back launches on the same inputs agree bit for bit and respect their buffers."""
    k = K()
    g = torch.Generator().manual_seed(3)
    logits = torch.randn(5, 151936, generator=g).to(DEV)
    buf = torch.full((5 + 16,), -7, dtype=torch.int64, device=DEV)
    a = k.argmax(logits, buf[8:13]).clone()
    b = k.argmax(logits, buf[8:13]).clone()
    assert torch.equal(a, b) and torch.equal(a.cpu(), logits.argmax(-1).cpu())
    assert bool((buf[:8] == -7).all()) and bool((buf[13:] == -7).all())
    nh, nkv, hd, rot, T = 8, 2, 64, 16, 300
    proj = bf(1, nh * 2 * hd + 2 * nkv * hd, seed=4).to(DEV)
    qg, kg = torch.ones(hd, device=DEV), torch.ones(hd, device=DEV)
    cos, sin = O.rope_tables(rot, 1e6, 512)
    kpool = bf(8 * 64, nkv, hd, seed=5).to(DEV)
    vpool = bf(8 * 64, nkv, hd, seed=6).to(DEV)
    bt = torch.arange(0, 8, dtype=torch.int32, device=DEV).reshape(1, -1)
    pos = torch.tensor([T], dtype=torch.int32, device=DEV)
    ns = k.decode_splits(nkv, 1)
    outs = []
    for _ in range(2):
        part_o = torch.zeros(1, nh, ns, hd, device=DEV)
        part_ml = torch.zeros(1, nh, ns, 2, device=DEV)
        tickets = torch.zeros(1, nkv, dtype=torch.int32, device=DEV)
        buf, out = _guarded(1, nh * hd, torch.bfloat16)
        k.attn_decode(proj, qg, kg, cos.to(DEV), sin.to(DEV), pos, pos, bt, kpool, vpool, part_o, part_ml, tickets, out,
                      nh=nh, nkv=nkv, hd=hd, rot=rot, nsplit=ns, eps=1e-6)
        torch.cuda.synchronize()
        assert _intact(buf, 1, nh * hd) and int(tickets.abs().sum()) == 0
        outs.append(out.clone())
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("M,N,Kd", [(2, 8, 8), (7, 136, 72), (16, 2560, 4096), (17, 12352, 2560), (33, 6176, 512), (64, 1000, 200),
                                    (65, 2048, 2048), (128, 40000, 264)])
def test_few_row_products(M, N, Kd):
    """Tile edges in rows (16 / 32 / 64 / 128) and columns, K tails, one slice and clusters of 2 to 8, one tile per CTA and several.
    Sums of bf16 products in fp32: 1e-5; one rounding to bf16 more: 2^-8 of the value.  int8: sums exact, scales in fp32."""
    k = K()
    from coffin_b200.ops import mixers as X
    A, W, res = bf(M, Kd, seed=1), bf(2 * N, Kd, s=Kd ** -0.5, seed=2), bf(M, N, seed=3)
    Ad, Wd = A.to(DEV), W.to(DEV)
    ref = A.to(DEV).double() @ Wd.double().t()
    g, u = ref[:, :N], ref[:, N:]

    def off(got, want):
        return ((got.double() - want).norm() / want.norm()).item()

    room = torch.full((M + 1, N + 8), 3.0, dtype=torch.bfloat16, device=DEV)
    assert off(k.gemm(Ad, Wd[:N], out=room[:M, :N], residual=res.to(DEV)), g + res.to(DEV).double()) < 4e-3
    assert bool((room[M] == 3.0).all()) and bool((room[:, N:] == 3.0).all())
    f = torch.full((M, N), float("nan"), device=DEV)
    assert off(k.gemm(Ad, Wd[:N], out=f), g) < 1e-5
    assert off(X.gemm_f32out(Ad, Wd[:N], f.fill_(float("nan"))), g) < 1e-5
    prod = torch.nn.functional.silu(g) * u
    assert off(k.gemm_swiglu(Ad, Wd), prod) < 4e-3
    main, gates = torch.empty(M, N, dtype=torch.bfloat16, device=DEV), torch.empty(M, N, device=DEV)
    X.gemm_mixed(Ad, Wd, main, gates)
    assert off(main, g) < 4e-3 and off(gates, u) < 1e-5
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    if M <= 8:                                       # decode projections of several rows end here too
        assert off(k.gemv(Wd, Ad, out, swiglu=True), prod) < 4e-3
        gain = torch.ones(Kd, device=DEV)
        h = k.rmsnorm(Ad, gain, 1e-6)
        assert off(k.gemv(Wd[:N], None, f, norm=(Ad, None, gain, None, 1e-6)), h.double() @ Wd[:N].double().t()) < 1e-5
    if Kd % 16 == 0:
        q, qs = k.quant_rows(Ad)
        w8, ws = k.quant_rows(Wd)
        r8 = (q.double() @ w8.double().t()) * qs.double()[:, None] * ws.double()
        assert off(k.gemm_i8(q, qs, w8[:N], ws[:N], out=f), r8[:, :N]) < 1e-6
        assert off(k.gemm_i8(q, qs, w8[:N], ws[:N], residual=res.to(DEV)), r8[:, :N] + res.to(DEV).double()) < 4e-3
        assert off(k.gemm_i8_swiglu(q, qs, w8, ws), torch.nn.functional.silu(r8[:, :N]) * r8[:, N:]) < 4e-3
        if M <= 8:
            assert off(k.gemv_i8(w8[:N], ws[:N], Ad, f), r8[:, :N]) < 1e-6


@pytest.mark.parametrize("M,N,Kd,kper", [(16, 2560, 4096, 22), (64, 2560, 9216, 21), (33, 264, 2048, 4), (64, 12352, 2560, 40), (9, 2048, 512, 4),
                                         (100, 1032, 4104, 9), (64, 2048, 4096, 16),
                                         (65, 12352, 520, 9), (128, 20000, 1024, 16)])
def test_few_row_products_keep_the_order_of_their_sums(M, N, Kd, kper):
    """Slices of ``kper`` k-blocks of 64, each summed along K and added in order, bit for bit: a slice by itself is a product of more than
    128 rows, which is not split.  (What follows in a model carries every change of rounding through all layers.)"""
    k = K()
    from coffin_b200.ops import mixers as X
    A, W = bf(160, Kd, seed=1).to(DEV), bf(N, Kd, s=Kd ** -0.5, seed=2).to(DEV)
    want, part = None, torch.empty(160, N, device=DEV)
    for at in range(0, Kd, 64 * kper):
        X.gemm_f32out(A[:, at:at + 64 * kper], W[:, at:at + 64 * kper], part)
        want = part.clone() if want is None else want + part
    assert torch.equal(X.gemm_f32out(A[:M], W, torch.empty(M, N, device=DEV)), want[:M])
    assert torch.equal(k.gemm(A[:M], W), want[:M].bfloat16())
    n = N // 16 * 8
    main, gates = torch.empty(M, n, dtype=torch.bfloat16, device=DEV), torch.empty(M, N - n, device=DEV)
    X.gemm_mixed(A[:M], W, main, gates)
    assert torch.equal(main, want[:M, :n].bfloat16()) and torch.equal(gates, want[:M, n:])


@pytest.mark.parametrize("M,I,Kd", [(1, 8, 64), (16, 9216, 2560), (64, 200, 520), (128, 1024, 2048)])
def test_few_row_swiglu_is_the_product_and_swiglu_after_it(M, I, Kd):
    """Gate and up are rounded to bf16 before the activation, bit for bit as two launches do it; int8 decode buckets leave both halves to
    the quantising kernel."""
    k = K()
    A, W = bf(M, Kd, seed=1).to(DEV), bf(2 * I, Kd, s=3 * Kd ** -0.5, seed=2).to(DEV)
    assert torch.equal(k.gemm_swiglu(A, W), k.swiglu(k.gemm(A, W)))
    if Kd % 16 == 0:
        from coffin_b200.models.qwen35.model import QW, Qwen35Model
        w = QW(*k.quant_rows(W))
        torch.cuda.synchronize()
        q, s = k.quant_rows(A)
        gu = torch.zeros(M, 2 * I, dtype=torch.bfloat16, device=DEV)
        assert object.__new__(Qwen35Model)._gemm_gu(A, w, gu, decode=True) is None
        assert torch.equal(gu, k.gemm_i8(q, s, w.wq, w.scale))


@pytest.mark.parametrize("M", [2, 128, 129, 300])
def test_products_store_the_type_of_their_result(M):
    """An fp32 result holds fp32 sums at any number of rows, a wider one keeps its other columns, and what has no such form is refused:
    the SwiGLU projections of decode rows, int8 products of more than 128 rows, a residual."""
    k = K()
    N, Kd = 264, 512
    A, W = bf(M, Kd, seed=1).to(DEV), bf(N, Kd, s=Kd ** -0.5, seed=2).to(DEV)
    ref = A.double() @ W.double().t()
    for out in (torch.full((M, N), 3.0, device=DEV), torch.full((M + 1, N + 8), 3.0, device=DEV)):
        k.gemm(A, W, out=out)
        assert ((out[:M, :N].double() - ref).norm() / ref.norm()).item() < 1e-5
        assert bool((out[M:] == 3.0).all()) and bool((out[:, N:] == 3.0).all())
    wide = torch.full((M, N + 8), 3.0, dtype=torch.bfloat16, device=DEV)
    assert torch.equal(k.gemm(A, W, out=wide)[:, :N], k.gemm(A, W)) and bool((wide[:, N:] == 3.0).all())
    f = torch.empty(M, N, device=DEV)
    refused = (AssertionError, k._lib.KernelError)
    with pytest.raises(refused):
        k.gemm(A, W, out=f, residual=torch.zeros(M, N, dtype=torch.bfloat16, device=DEV))
    q8, w8 = k.quant_rows(A), k.quant_rows(W)
    if M > 128:
        with pytest.raises(refused):
            k.gemm_i8(*q8, *w8, out=f)
    else:
        with pytest.raises(refused):
            k.gemm(A, W, out=wide[:, :N - 8])
        k.gemm_i8(*q8, *w8, out=f)
        want = (q8[0].double() @ w8[0].double().t()) * q8[1].double()[:, None] * w8[1].double()
        assert ((f.double() - want).norm() / want.norm()).item() < 1e-6
    if M <= 8:
        half = torch.empty(M, N // 2, device=DEV)
        with pytest.raises(refused):
            k.gemv(W, A, half, swiglu=True)
        with pytest.raises(refused):
            k.gemv_i8(*w8, A, half, swiglu=True)
    else:                                            # decode projections take up to eight rows
        b = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        with pytest.raises(refused):
            k.gemv(W, A, b)
        with pytest.raises(refused):
            k.gemv_i8(*w8, A, b)


@pytest.mark.parametrize("M", [2, 8, 100])
def test_int8_products_of_few_rows_take_scales_from_anywhere(M):
    """Rows [1:] of a weight have their scales 4 bytes behind a vector's border, as slices of an int8 projection do."""
    k = K()
    N, Kd = 264, 512
    A, W = bf(M, Kd, seed=1).to(DEV), bf(2 * N + 1, Kd, s=Kd ** -0.5, seed=2).to(DEV)
    wq, ws = k.quant_rows(W)
    a8 = k.quant_rows(A)
    part, scale = wq[1:].contiguous(), ws[1:].clone()
    torch.cuda.synchronize()
    assert ws[1:].data_ptr() % 16 == 4
    assert torch.equal(k.gemm_i8(*a8, part, ws[1:]), k.gemm_i8(*a8, part, scale))
    assert torch.equal(k.gemm_i8_swiglu(*a8, part, ws[1:]), k.gemm_i8_swiglu(*a8, part, scale))
    if M <= 8:
        outs = [torch.empty(M, 2 * N, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
        assert torch.equal(*(k.gemv_i8(part, s, A, o) for s, o in zip((ws[1:], scale), outs)))
        outs = [o[:, :N].contiguous() for o in outs]
        assert torch.equal(*(k.gemv_i8(part, s, A, o, swiglu=True) for s, o in zip((ws[1:], scale), outs)))
    off = torch.empty(M * N + 1, device=DEV)[1:].view(M, N)
    with pytest.raises(k._lib.KernelError):          # results travel by fours
        k.gemm(A, W[:N], out=off)


def test_few_row_products_of_weights_just_written():
    """The second operand written by the launch right in front, or by the one before that, into a block that held other values: int4
    expansions (resident after ``settle``, or not said to be resident), quantised rows, rows of another product."""
    k = K()
    from coffin_b200.ops import mixers as X
    from coffin_b200.weights.quant import W4A8Weight
    M, N, Kd, turns = 24, 4096, 2560, 6
    A = bf(M, Kd, seed=1).to(DEV)
    codes = [tuple(t.to(DEV) for t in W4A8Weight.quantize(bf(N, Kd, seed=10 + i).float() * 0.1).to_nk()) for i in range(turns)]
    plain = [bf(N, Kd, seed=30 + i).to(DEV) for i in range(turns)]
    near = [bf(N, 512, seed=50 + i).to(DEV) for i in range(turns)]
    low = bf(Kd, 512, seed=70, s=0.05).to(DEV)
    W, f32 = torch.empty(N, Kd, dtype=torch.bfloat16, device=DEV), torch.empty(M, N, device=DEV)
    res = []
    for wait in (True, False):
        sync = torch.cuda.synchronize if wait else (lambda: None)
        outs = []
        for i in range(turns):
            sync()
            k.w4_dequant(*codes[i], out=W)
            sync()
            outs.append(k.gemm(A, W))
            sync()
            k.w4_dequant(*codes[-1 - i], out=W)
            k.settle()
            outs.append(k.gemm(A, W, resident=True))
            sync()
            q8 = k.quant_rows(plain[i])
            a8 = k.quant_rows(A)
            sync()
            outs += [k.gemm_i8(*a8, *q8), k.gemm_i8_swiglu(*a8, *q8)]
            sync()
            k.gemm(near[i], low, out=W)
            sync()
            outs.append(X.gemm_f32out(A, W, f32).clone())
            sync()
            k.gemm(near[-1 - i], low, out=W)
            sync()
            outs.append(k.gemm_swiglu(A, W))
            sync()
            k.gemm(near[i], low, out=W)
            sync()
            outs.append(X.linear_xielu(W, A, torch.empty(M, N, dtype=torch.bfloat16, device=DEV), 0.8, 0.9))
            main, gates = torch.empty(M, N - 64, dtype=torch.bfloat16, device=DEV), torch.empty(M, 64, device=DEV)
            k.gemm(near[-1 - i], low, out=W)
            sync()
            X.gemm_mixed(A, W, main, gates)
            outs += [main, gates]
        torch.cuda.synchronize()
        res.append(outs)
    for i, (x, y) in enumerate(zip(*res)):
        assert torch.equal(x, y), i


@pytest.mark.parametrize("nk,nv,dk,lens", [(16, 32, 128, (1, 64, 65, 130, 300)), (16, 48, 128, (512, 127)), (2, 4, 64, (3, 200, 64))])
def test_gdn_prefill_of_several_sequences(nk, nv, dk, lens):
    """One call over stacked sequences against one call each, bit for bit: chunk edges, a slot order of its own, rows before the
    chunk from the ring, value heads of a key head in one CTA (from 148 (chunk, key head) pairs on) or one each."""
    k = K()
    T, n = sum(lens), len(lens)
    proj, conv_w, A_log, dt_bias, norm_w, conv_dim = _gdn_inputs(T, nk, nv, dk, dk, 77)
    d = lambda t: t.to(DEV)
    g = torch.Generator().manual_seed(78)
    ring = torch.randn(n + 1, k.RING, conv_dim, generator=g).bfloat16().to(DEV)
    st = (0.1 * torch.randn(n + 1, nv, dk, dk, generator=g)).to(DEV)
    args = (d(conv_w), d(A_log), d(dt_bias), d(norm_w.float()))
    kw = dict(nk=nk, nv=nv, dk=dk, dv=dk, eps=1e-6)
    pj, segs = d(proj), [(m, 5 * i, (i + 2) % (n + 1)) for i, m in enumerate(lens)]
    r2, s2, want = ring.clone(), st.clone(), torch.empty(T, nv * dk, dtype=torch.bfloat16, device=DEV)
    scratch = torch.empty(k.gdn_prefill_scratch_floats(T, nk, nv, dk, dk, n), device=DEV)
    at = 0
    for m, pos, slot in segs:
        k.gdn_prefill(pj[at:at + m], *args, r2[slot], s2[slot], scratch, want[at:at + m], pos0=pos, **kw)
        at += m
    got = torch.empty_like(want)
    k.gdn_prefill_group(pj, *args, ring, st, scratch.fill_(float("nan")), got, segs, **kw)
    assert torch.equal(got, want) and torch.equal(ring, r2) and torch.equal(st, s2)


@pytest.mark.parametrize("hd,lens", [(64, (32, 31, 129, 1, 500)), (256, (128, 40, 200))])
def test_attention_of_several_sequences(hd, lens):
    """One launch for the sequences of at least 32 rows (query tiles of 128) against one call per sequence, bit for bit."""
    k = K()
    nh, nkv, T = 4, 2, sum(lens)
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)
    before = [70 * i for i in range(len(lens))]
    pages = [(b + m + 63) // 64 for b, m in zip(before, lens)]
    order = torch.randperm(sum(pages), generator=g).to(torch.int32).to(DEV)
    kpool, vpool = rnd(sum(pages) * 64, nkv, hd), rnd(sum(pages) * 64, nkv, hd)
    q, proj = rnd(T, nh, hd), rnd(T, nh * 2 * hd)
    segs, at, pg = [], 0, 0
    want, got = torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV), torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV)
    for m, b, p in zip(lens, before, pages):
        bt = order[pg:pg + p].clone()
        segs.append((at, m, b, bt))
        k.attn_prefill(q[at:at + m], proj[at:at + m], kpool, vpool, bt, want[at:at + m], q_pos0=b, nh=nh, nkv=nkv, hd=hd)
        at, pg = at + m, pg + p
    k.attn_prefill_group(q, proj, kpool, vpool, got, segs, nh=nh, nkv=nkv, hd=hd)
    assert torch.equal(got, want)


@pytest.mark.parametrize("nk,nv,M", [(16, 32, 10), (16, 48, 64), (5, 5, 61)])
def test_gdn_decode_of_many_rows(nk, nv, M):
    """More (row, head) pairs than two CTAs an SM hold: the streaming kernel against the per-pair one on eight rows at a time.  The
    norm's sum is taken in another order (fp32, one bf16 rounding) and the compiler contracts other multiplies and adds: a few fp32
    roundings (2^-24 each) of sums of 128 terms, 1e-5 of the scale.  Padded rows stay untouched."""
    k = K()
    dk, n = 128, M + 2
    proj, conv_w, A_log, dt_bias, norm_w, conv_dim = _gdn_inputs(M, nk, nv, dk, dk, 91)
    g = torch.Generator().manual_seed(92)
    ring = torch.randn(n, k.RING, conv_dim, generator=g).bfloat16().to(DEV)
    st = (0.1 * torch.randn(n, nv, dk, dk, generator=g)).to(DEV)
    slots = torch.randperm(n, generator=g)[:M].to(torch.int32)
    slots[3] = slots[M - 1] = -1
    pos = torch.randint(0, 40, (M,), generator=g, dtype=torch.int32)
    slots, pos, pj = slots.to(DEV), pos.to(DEV), proj.to(DEV)
    args = [t.to(DEV) for t in (conv_w, A_log, dt_bias, norm_w.float())]
    kw = dict(nk=nk, nv=nv, dk=dk, dv=dk, eps=1e-6)
    r2, s2, want, got = ring.clone(), st.clone(), torch.zeros(M, nv * dk, dtype=torch.bfloat16, device=DEV), torch.zeros(M, nv * dk, dtype=torch.bfloat16, device=DEV)
    step = max(1, min(8, 290 // nv))
    for at in range(0, M, step):
        sl = slice(at, at + step)
        k.gdn_decode(pj[sl], *args, r2, s2, slots[sl].contiguous(), pos[sl].contiguous(), want[sl], **kw)
    k.gdn_decode(pj, *args, ring, st, slots, pos, got, **kw)
    k.check_status()
    assert torch.equal(ring, r2)
    close(st, s2, 1e-5)
    close(got, want, 2 ** -7)


@pytest.mark.parametrize("nk,nv,M", [(16, 32, 64), (16, 48, 17), (5, 5, 61)])
def test_gdn_decode_of_many_rows_is_that_of_few(nk, nv, M):
    """A row's state, ring and output are the same bits whether it steps with many rows or with few (states of ordinary size, three
    steps, first tokens among them)."""
    k = K()
    dk = 128
    conv_dim = 2 * nk * dk + nv * dk
    g = torch.Generator().manual_seed(93)
    ring, st = torch.zeros(M, k.RING, conv_dim, dtype=torch.bfloat16, device=DEV), torch.zeros(M, nv, dk, dk, device=DEV)
    st[::2] = (0.1 * torch.randn(st[::2].shape, generator=g)).to(DEV)
    slots = torch.randperm(M, generator=g).to(torch.int32).to(DEV)
    _, conv_w, A_log, dt_bias, norm_w, _ = _gdn_inputs(M, nk, nv, dk, dk, 94)
    args = [t.to(DEV) for t in (conv_w, A_log, dt_bias, norm_w.float())]
    kw = dict(nk=nk, nv=nv, dk=dk, dv=dk, eps=1e-6)
    r2, s2, few = ring.clone(), st.clone(), 290 // nv if nv < 290 else 1
    for step in range(3):
        pj = _gdn_inputs(M, nk, nv, dk, dk, 95 + step)[0].to(DEV)
        pos = torch.full((M,), step, dtype=torch.int32, device=DEV)
        want, got = (torch.zeros(M, nv * dk, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        torch.cuda.synchronize()
        for at in range(0, M, few):
            sl = slice(at, at + few)
            k.gdn_decode(pj[sl], *args, r2, s2, slots[sl].contiguous(), pos[sl].contiguous(), want[sl], **kw)
        torch.cuda.synchronize()
        k.gdn_decode(pj, *args, ring, st, slots, pos, got, **kw)
        torch.cuda.synchronize()
        assert torch.equal(st, s2) and torch.equal(ring, r2) and torch.equal(got, want), step


@pytest.mark.parametrize("M", [4, 40])
def test_gdn_decode_steps_that_follow_one_another(M):
    """Steps enqueued back to back on one state, with nothing between them (the step before may still run when one starts), and a
    commit of recorded tokens in front: the same bits as with the device waited for after every launch."""
    k = K()
    nk, nv, dk, ntok, steps = 16, 32, 128, 2, 12
    g = torch.Generator().manual_seed(7)
    _, conv_w, A_log, dt_bias, norm_w, conv_dim = _gdn_inputs(M, nk, nv, dk, dk, 96)
    args = [t.to(DEV) for t in (conv_w, A_log, dt_bias, norm_w.float())]
    kw = dict(nk=nk, nv=nv, dk=dk, dv=dk, eps=1e-6)
    pjs = [_gdn_inputs(M, nk, nv, dk, dk, 100 + i)[0].to(DEV) for i in range(steps)]
    pair = _gdn_inputs(M * ntok, nk, nv, dk, dk, 99)[0].to(DEV)
    slots, pos = torch.randperm(M, generator=g).to(torch.int32).to(DEV), torch.zeros(M, dtype=torch.int32, device=DEV)
    ring0 = torch.randn(M, k.RING, conv_dim, generator=g).bfloat16().to(DEV)
    st0 = (0.1 * torch.randn(M, nv, dk, dk, generator=g)).to(DEV)
    record = torch.zeros(M, ntok, nv * (2 * dk + 1), device=DEV)
    accept = torch.full((M,), ntok, dtype=torch.int32, device=DEV)
    at = [pos + ntok + i for i in range(steps)]
    res = []
    for wait in (True, False):
        ring, st = ring0.clone(), st0.clone()
        outs = [torch.zeros(M, nv * dk, dtype=torch.bfloat16, device=DEV) for _ in range(steps)]
        sync = torch.cuda.synchronize if wait else (lambda: None)
        torch.cuda.synchronize()
        k.gdn_decode(pair, *args, ring, st, slots, pos, torch.empty(M * ntok, nv * dk, dtype=torch.bfloat16, device=DEV), ntok=ntok,
                     record=record, write_state=False, **kw)
        sync()
        k.gdn_commit(st, record, slots, accept, nv=nv, dk=dk, dv=dk)
        sync()
        for i in range(steps):
            k.gdn_decode(pjs[i], *args, ring, st, slots, at[i], outs[i], **kw)
            sync()
        torch.cuda.synchronize()
        k.check_status()
        res.append((ring, st, *outs))
    assert all(torch.equal(x, y) for x, y in zip(*res))


@pytest.mark.parametrize("E,N,Kd,swiglu,slots", [(6, 128, 256, True, 97), (5, 520, 2304, False, 200), (300, 24, 128, True, 512), (3, 2048, 512, False, 1024)])
def test_moe_gemv_w4a8_by_expert(E, N, Kd, swiglu, slots, monkeypatch):
    """Experts taken whole (several passes of eight slots, experts without a slot, slots of other ranks, row and K remainders) against
    the slot-wise kernel: the same integers and scales, fp32 sums of at most 18 groups in another order, one bf16 rounding."""
    k = K()
    from coffin_b200.weights.quant import W4A8Weight
    g = torch.Generator().manual_seed(70)
    W = torch.randn(E, 2 * N if swiglu else N, Kd, generator=g) * 0.05
    wq, sc = (t.to(DEV) for t in W4A8Weight.quantize(W).to_nk())
    x = torch.randn(slots, Kd, generator=g).bfloat16().to(DEV)
    slot_e = torch.randint(-1, max(1, E * 2 // 3), (slots,), generator=g, dtype=torch.int32).to(DEV)
    slot_x = torch.randint(0, slots, (slots,), generator=g, dtype=torch.int32).to(DEV)
    for rows in (slot_x, None):
        want, got = (torch.full((slots, N), 3.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        monkeypatch.setattr(k, "W4_GROUP_SHARE", 1 << 20)
        k.moe_gemv_w4(wq, sc, x, want, slot_e, rows, swiglu=swiglu)
        monkeypatch.setattr(k, "W4_GROUP_SHARE", 0)
        k.moe_gemv_w4(wq, sc, x, got, slot_e, rows, swiglu=swiglu)
        assert bool((got[slot_e < 0] == 3.0).all())
        close(got, want, 2 ** -7)


@pytest.mark.parametrize("E,T,kind", [(256, 33, "padded"), (256, 64, "wanted"), (600, 64, "padded"), (2, 128, "wanted"), (7, 9, "one")])
def test_moe_gemv_w4a8_by_expert_of_uneven_routing(E, T, kind, monkeypatch):
    """Passes of eight slots of one expert in CTAs of their own: the rows behind the last sequence all alike, experts that every row wants
    (9, 64 and 65 slots), all slots on one expert, one after it; every slot's result that of the slot-wise kernel, twice the same bits."""
    k = K()
    from coffin_b200.weights.quant import W4A8Weight
    g = torch.Generator().manual_seed(E + T)
    top = min(8, E)
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    if kind == "padded":
        idx[T // 2:] = idx[-1]
    elif kind == "wanted":
        idx[:, 0] = E - 1
        idx[:min(T, 9), 1] = 0
    else:
        idx[:] = E - 2
    N, Kd = 40, 256
    wq, sc = (t.to(DEV) for t in W4A8Weight.quantize(torch.randn(E, N, Kd, generator=g) * 0.05).to_nk())
    x = torch.randn(T, Kd, generator=g).bfloat16().to(DEV)
    slots, rows = idx.reshape(-1).contiguous().to(DEV), torch.arange(T, dtype=torch.int32, device=DEV).repeat_interleave(top).contiguous()
    want, got = (torch.full((T * top, N), 3.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    monkeypatch.setattr(k, "W4_GROUP_SHARE", 1 << 20)
    k.moe_gemv_w4(wq, sc, x, want, slots, rows)
    monkeypatch.setattr(k, "W4_GROUP_SHARE", 0)
    k.moe_gemv_w4(wq, sc, x, got, slots, rows)
    close(got, want, 2 ** -7)
    assert torch.equal(k.moe_gemv_w4(wq, sc, x, torch.full_like(got, 3.0), slots, rows), got)


@pytest.mark.parametrize("M,nkv,nsplit", [(8, 4, 64), (9, 4, 1), (16, 2, 2), (70, 1, 9)])
def test_decode_attention_of_rows_of_any_length(M, nkv, nsplit):
    """Tiles of all rows shared evenly (runs that start and end inside a row, whole pairs when there is room for one partial, padded
    rows, a first token) against the kernel that takes a row at a time: scores and sums in fp32, P rounded to bf16 in one of them."""
    k = K()
    rep, hd, rot = 4, 256, 64
    nh = nkv * rep
    g = torch.Generator().manual_seed(M)
    pos = torch.randint(0, 900, (M,), generator=g, dtype=torch.int32)
    pos[0], pos[1], pos[M // 2], pos[M - 1] = 0, 3001, -1, 63
    pages = [(int(p) + 64) // 64 for p in pos.clamp(min=0)]
    order, bt, at = torch.randperm(sum(pages), generator=g), torch.zeros(M, max(pages), dtype=torch.int32), 0
    for m, p in enumerate(pages):
        bt[m, :p] = order[at:at + p]
        at += p
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)
    kp, vp = rnd(sum(pages) * 64, nkv, hd), rnd(sum(pages) * 64, nkv, hd)
    proj = rnd(M, nh * 2 * hd + 2 * nkv * hd)
    gain = torch.ones(hd, device=DEV)
    cos, sin = O.rope_tables(rot, 1e6, 3100)
    pos, bt, cos, sin = pos.to(DEV), bt.to(DEV), cos.to(DEV), sin.to(DEV)

    def run(ctas, ns):
        pools, out = (kp.clone(), vp.clone()), torch.zeros(M, nh * hd, dtype=torch.bfloat16, device=DEV)
        part_o, part_ml = torch.empty(M, nh, ns, hd, device=DEV), torch.empty(M, nh, ns, 2, device=DEV)
        tickets = torch.zeros(M, nkv, dtype=torch.int32, device=DEV)
        k._lib.call_nostream("set_attn_batch_ctas", ctas)
        try:
            for _ in range(2):
                k.attn_decode(proj, gain, gain, cos, sin, pos, pos.clamp(min=0), bt, *pools, part_o, part_ml, tickets, out, nh=nh, nkv=nkv,
                              hd=hd, rot=rot, nsplit=ns, eps=1e-6)
        finally:
            k._lib.call_nostream("set_attn_batch_ctas", 32)
        assert not bool(tickets.any())
        return out, pools

    (want, wp), (got, gp) = run(0, 8), run(1, nsplit)
    assert torch.equal(wp[0], gp[0]) and torch.equal(wp[1], gp[1])
    close(got, want, 1e-2)


@pytest.mark.parametrize("M,nkv", [(16, 4), (33, 2), (64, 4), (130, 1)])
def test_decode_attention_of_wide_batches_takes_a_row_by_itself(M, nkv):
    """From nine rows on a row's output is the same bits whatever the lengths of the others, with one split a row and several, splits
    without a tile, and the row's token in the last one; a second run repeats them."""
    k = K()
    rep, hd, rot = 4, 256, 64
    nh, ns = nkv * rep, k.decode_splits(nkv, M)
    g = torch.Generator().manual_seed(M)
    bt = torch.randperm(M * 20, generator=g).to(torch.int32).view(M, 20).to(DEV)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)
    kp, vp = rnd(M * 20 * 64, nkv, hd), rnd(M * 20 * 64, nkv, hd)
    proj = rnd(M, nh * 2 * hd + 2 * nkv * hd)
    gain = torch.ones(hd, device=DEV)
    cos, sin = (t.to(DEV) for t in O.rope_tables(rot, 1e6, 1300))
    one = torch.randint(0, 1280, (M,), generator=g, dtype=torch.int32)
    one[:3] = torch.tensor([0, 63, 1279])
    two = torch.randint(0, 1280, (M,), generator=g, dtype=torch.int32)
    two[:M // 2] = one[:M // 2]
    outs = []
    for pos in (one, two):
        pos, pools, out = pos.to(DEV), (kp.clone(), vp.clone()), torch.zeros(M, nh * hd, dtype=torch.bfloat16, device=DEV)
        part_o, part_ml = torch.empty(M, nh, ns, hd, device=DEV), torch.empty(M, nh, ns, 2, device=DEV)
        tickets = torch.zeros(M, nkv, dtype=torch.int32, device=DEV)
        for turn in range(2):
            before = out.clone()
            if turn:                                 # pools may come as blocks of rows
                pools = [t.view(-1, 64, nkv, hd) for t in pools]
            k.attn_decode(proj, gain, gain, cos, sin, pos, pos, bt, *pools, part_o, part_ml, tickets, out, nh=nh, nkv=nkv, hd=hd, rot=rot,
                          nsplit=ns, eps=1e-6)
        assert torch.equal(out, before)
        outs.append(out[:M // 2])
    assert torch.equal(*outs)


@pytest.mark.parametrize("M,nkv,nsplit", [(8, 4, 64), (9, 4, 1), (16, 2, 4), (70, 1, 9)])
def test_decode_attention_of_int8_pages(M, nkv, nsplit):
    """The batch kernel on int8 pages (rows of one token, of a tile and one more, several tiles a split and none, padded rows) against the
    kernel that takes a row at a time: the pages and scales it writes are the same bytes; scores and sums in fp32, keys and values
    rounded to bf16 (2^-9) in both, P in one of them.  A second run gives the same bits."""
    k = K()
    rep, hd, rot = 4, 256, 64
    nh = nkv * rep
    g = torch.Generator().manual_seed(M)
    pos = torch.randint(0, 900, (M,), generator=g, dtype=torch.int32)
    pos[0], pos[1], pos[2], pos[3], pos[M // 2], pos[M - 1] = 0, 3001, 64, 127, -1, 63
    pages = [(int(p) + 64) // 64 for p in pos.clamp(min=0)]
    order, bt, at = torch.randperm(sum(pages), generator=g), torch.zeros(M, max(pages), dtype=torch.int32), 0
    for m, p in enumerate(pages):
        bt[m, :p] = order[at:at + p]
        at += p
    rows = sum(pages) * 64
    q8 = [torch.randint(-127, 128, (rows, nkv, hd), generator=g, dtype=torch.int8).to(DEV) for _ in range(2)]
    sc = [(torch.rand(rows, nkv, generator=g) * 0.02 + 0.005).to(DEV) for _ in range(2)]
    proj = torch.randn(M, nh * 2 * hd + 2 * nkv * hd, generator=g).bfloat16().to(DEV)
    gain = torch.ones(hd, device=DEV)
    cos, sin = (t.to(DEV) for t in O.rope_tables(rot, 1e6, 3100))
    pos, bt = pos.to(DEV), bt.to(DEV)

    def run(ctas, ns):
        pools, scales, out = [t.clone() for t in q8], [t.clone() for t in sc], torch.zeros(M, nh * hd, dtype=torch.bfloat16, device=DEV)
        part_o, part_ml = torch.empty(M, nh, ns, hd, device=DEV), torch.empty(M, nh, ns, 2, device=DEV)
        tickets = torch.zeros(M, nkv, dtype=torch.int32, device=DEV)
        k._lib.call_nostream("set_attn_batch_ctas", ctas)
        try:
            for _ in range(2):
                before = out.clone()
                k.attn_decode(proj, gain, gain, cos, sin, pos, pos.clamp(min=0), bt, *pools, part_o, part_ml, tickets, out, nh=nh, nkv=nkv,
                              hd=hd, rot=rot, nsplit=ns, eps=1e-6, kscale=scales[0], vscale=scales[1])
        finally:
            k._lib.call_nostream("set_attn_batch_ctas", 32)
        assert not bool(tickets.any()) and torch.equal(before, out)
        return out, pools, scales

    (want, wp, ws), (got, gp, gs) = run(0, 8), run(1, nsplit)
    assert all(torch.equal(x, y) for x, y in zip(wp + ws, gp + gs))
    close(got, want, 1e-2)
