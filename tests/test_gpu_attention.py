"""GPU parity of the decode-step neighbours: fused split + qk-norm + RoPE + KV write, and paged attention."""
import numpy as np
import pytest
import torch

from oracle import fishref

pytestmark = pytest.mark.gpu

N_Q, N_KV, D, LAYERS, BS = 32, 8, 128, 3, 16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def make_cache(rng, B, ctx_len, max_blocks):
    nblk = B * max_blocks + 3
    kc = (rng.standard_normal((nblk, LAYERS, N_KV, BS, D)) * 0.5).astype(np.float16)
    vc = (rng.standard_normal((nblk, LAYERS, N_KV, BS, D)) * 0.5).astype(np.float16)
    perm = rng.permutation(nblk)[:B * max_blocks].reshape(B, max_blocks).astype(np.int32)  # scattered physical blocks
    return kc, vc, perm


@pytest.mark.parametrize("B,with_norm", [(1, True), (8, True), (3, False)])
def test_qknorm_rope_kvwrite(ctx, oracle, B, with_norm):
    rng = np.random.default_rng(B)
    layer, max_blocks = 1, 8
    qkv = rng.standard_normal((B, (N_Q + 2 * N_KV) * D)).astype(np.float16)
    qw = rng.uniform(0.5, 1.5, D).astype(np.float16)
    kw = rng.uniform(0.5, 1.5, D).astype(np.float16)
    freqs = oracle.rope_freqs(D, 1e6)
    positions = rng.integers(0, max_blocks * BS, B).astype(np.int32)
    kc, vc, bt = make_cache(rng, B, 0, max_blocks)
    dk, dv = dev(kc), dev(vc)
    dq = torch.empty((B, N_Q, D), dtype=torch.float16, device="cuda")
    dqkv, dqw, dkw, dfr, dpos, dbt = dev(qkv), dev(qw), dev(kw), dev(freqs), dev(positions), dev(bt)
    ctx.qknorm_rope_kvwrite(dqkv, dqw if with_norm else None, dkw if with_norm else None, 1e-6, dfr, dpos, dbt,
                            max_blocks, dk, dv, layer, LAYERS, B, N_Q, N_KV, D, dq)
    torch.cuda.synchronize()
    q3 = qkv.reshape(B, N_Q + 2 * N_KV, D)
    want_k, want_v = kc.copy(), vc.copy()
    for b in range(B):
        pos = int(positions[b])
        wq = oracle.qknorm_rope(q3[b, :N_Q], qw if with_norm else None, 1e-6, freqs, pos)
        wk = oracle.qknorm_rope(q3[b, N_Q:N_Q + N_KV], kw if with_norm else None, 1e-6, freqs, pos)
        assert oracle.ulp_distance_fp16(dq[b].cpu().numpy(), wq).max() <= 2
        phys = bt[b, pos // BS]
        got_k = dk[phys, layer, :, pos % BS].cpu().numpy()
        assert oracle.ulp_distance_fp16(got_k, wk).max() <= 2
        want_k[phys, layer, :, pos % BS] = got_k
        want_v[phys, layer, :, pos % BS] = q3[b, N_Q + N_KV:]
    # nothing but the B new rows changed, and v is a verbatim copy
    assert np.array_equal(dk.cpu().numpy(), want_k) and np.array_equal(dv.cpu().numpy(), want_v)
    if fishref.available():
        # the reference chain: rms_norm on q and k, rope_qk in place (one sequence at a time: it is batch-1 code)
        for b in range(B):
            rq, rk = dev(q3[b, :N_Q].copy()), dev(q3[b, N_Q:N_Q + N_KV].copy())
            if with_norm:
                fishref.rms_norm(rq.data_ptr(), dqw.data_ptr(), rq.data_ptr(), N_Q, D, 1e-6)
                fishref.rms_norm(rk.data_ptr(), dkw.data_ptr(), rk.data_ptr(), N_KV, D, 1e-6)
            fishref.rope_qk(rq.data_ptr(), rk.data_ptr(), dfr.data_ptr(), 1, N_Q, N_KV, 1, D, int(positions[b]))
            torch.cuda.synchronize()
            assert torch.equal(rq, dq[b]), "q must match the reference chain bit for bit"
            pos = int(positions[b])
            assert torch.equal(rk, dk[int(bt[b, pos // BS]), layer, :, pos % BS])


@pytest.mark.parametrize("B,lens", [(1, [1]), (2, [16, 17]), (8, [1024] * 8), (4, [5, 300, 0, 1000])])
@pytest.mark.parametrize("splits", [0, 1, 3])
def test_paged_attention_decode(ctx, oracle, B, lens, splits):
    rng = np.random.default_rng(B + len(lens))
    layer, max_blocks = 2, 128
    kc, vc, bt = make_cache(rng, B, max(lens), max_blocks)
    q = rng.standard_normal((B, N_Q, D)).astype(np.float16)
    seq = np.array(lens, np.int32)
    dq, dk, dv, dbt, dseq = dev(q), dev(kc), dev(vc), dev(bt), dev(seq)
    dout = torch.full((B, N_Q, D), 9.0, dtype=torch.float16, device="cuda")
    sm = 1.0 / np.sqrt(D)
    for g in (256, 64):
        dxq = torch.empty((B, N_Q * D), dtype=torch.int8, device="cuda")
        dxs = torch.empty((B, N_Q * D // g), dtype=torch.float32, device="cuda")
        ctx.paged_attention_decode(dq, dk, dv, dbt, dseq, dout, B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV,
                                   quant_group_size=g, Xq=dxq, Xs=dxs, context_splits=splits)
        torch.cuda.synchronize()
        got = dout.cpu().numpy()
        want = oracle.paged_attention_decode(q, kc, vc, bt, seq, layer, sm)
        assert np.abs(got.astype(np.float64) - want).max() <= 2e-3 * max(1.0, np.abs(want).max())
        # the fused quantiser == the stand-alone quantiser on the fp16 output
        wq, ws = oracle.quantize(got.reshape(B, N_Q * D), g)
        assert np.array_equal(dxq.cpu().numpy(), wq) and np.array_equal(dxs.cpu().numpy(), ws)
    if fishref.available():
        rout = torch.empty_like(dout)
        fishref.paged_attention_decode(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dbt.data_ptr(), dseq.data_ptr(),
                                       rout.data_ptr(), B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV)
        torch.cuda.synchronize()
        assert (rout.float() - dout.float()).abs().max().item() <= 2e-3 * max(1.0, rout.float().abs().max().item())


# One to eight slices as the launch chooses them (the table's width and the batch decide), the longest sequence filling the table.
@pytest.mark.parametrize("B,max_blocks", [(8, 25), (1, 26), (8, 26), (1, 44), (5, 45), (3, 40), (4, 128), (2, 128), (1, 128), (10, 128), (8, 60)])
def test_paged_attention_decode_with_chosen_slices(ctx, oracle, B, max_blocks):
    rng = np.random.default_rng(B + max_blocks)
    layer = 1
    lens = [max_blocks * BS] + [int(rng.integers(0, max_blocks * BS)) for _ in range(B - 1)]
    kc, vc, bt = make_cache(rng, B, max(lens), max_blocks)
    q = rng.standard_normal((B, N_Q, D)).astype(np.float16)
    seq = np.array(lens, np.int32)
    dout = torch.full((B, N_Q, D), 9.0, dtype=torch.float16, device="cuda")
    sm = 1.0 / np.sqrt(D)
    ctx.paged_attention_decode(dev(q), dev(kc), dev(vc), dev(bt), dev(seq), dout, B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV)
    torch.cuda.synchronize()
    ctx.check_device_status()
    want = oracle.paged_attention_decode(q, kc, vc, bt, seq, layer, sm)
    assert np.abs(dout.cpu().numpy().astype(np.float64) - want).max() <= 2e-3 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("B,positions", [(1, [0]), (3, [15, 16, 40]), (8, [1024] * 8), (4, [4, 299, 31, 999])])
@pytest.mark.parametrize("splits", [0, 1, 2, 3])
def test_qkv_attention_decode_equals_the_two_calls(ctx, B, positions, splits):
    """qk-norm + RoPE + KV write + attention (+ quantiser) as one launch against the two launches: attention
    output, codes, scales and both caches bit for bit."""
    rng = np.random.default_rng(B + sum(positions))
    layer, max_blocks, g = 1, 128, 256
    kc, vc, bt = make_cache(rng, B, max(positions) + 1, max_blocks)
    qkv = rng.standard_normal((B, (N_Q + 2 * N_KV) * D)).astype(np.float16)
    qw = rng.uniform(0.5, 1.5, D).astype(np.float16)
    kw = rng.uniform(0.5, 1.5, D).astype(np.float16)
    freqs = (1.0 / np.power(np.float32(1e6), np.float32(2.0) * np.arange(D // 2, dtype=np.float32) / np.float32(D))
             ).astype(np.float32)
    pos = np.array(positions, np.int32)
    dqkv, dqw, dkw, dfr, dpos, dbt = dev(qkv), dev(qw), dev(kw), dev(freqs), dev(pos), dev(bt)
    dseq = dev(pos + 1)
    sm = 1.0 / np.sqrt(D)

    def run(fused):
        dk, dv = dev(kc), dev(vc)
        out = torch.full((B, N_Q, D), 7.0, dtype=torch.float16, device="cuda")
        xq = torch.full((B, N_Q * D), 99, dtype=torch.int8, device="cuda")
        xs = torch.full((B, N_Q * D // g), -1.0, dtype=torch.float32, device="cuda")
        if fused:
            ctx.qkv_attention_decode(dqkv, dqw, dkw, 1e-6, dfr, dpos, dk, dv, dbt, dseq, out, B, N_Q, D, max_blocks, sm,
                                     layer, LAYERS, N_KV, quant_group_size=g, Xq=xq, Xs=xs, context_splits=splits)
        else:
            dq = torch.empty((B, N_Q, D), dtype=torch.float16, device="cuda")
            ctx.qknorm_rope_kvwrite(dqkv, dqw, dkw, 1e-6, dfr, dpos, dbt, max_blocks, dk, dv, layer, LAYERS, B, N_Q, N_KV,
                                    D, dq)
            ctx.paged_attention_decode(dq, dk, dv, dbt, dseq, out, B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV,
                                       quant_group_size=g, Xq=xq, Xs=xs, context_splits=splits)
        torch.cuda.synchronize()
        return out, xq, xs, dk, dv

    want, got = run(False), run(True)
    for w, gt, what in zip(want, got, ("attention output", "codes", "scales", "k cache", "v cache")):
        assert torch.equal(w.view(torch.uint8) if w.dtype != torch.int8 else w, gt.view(torch.uint8) if gt.dtype != torch.int8 else gt), what
    assert not torch.equal(got[3], dev(kc)), "the new k rows were written"


def chained_setup(oracle, B, context, steps, max_blocks):
    """`steps` consecutive tokens of one layer: their qkv rows, positions and lengths, all on the device before the first call."""
    rng = np.random.default_rng(context + steps)
    kc, vc, bt = make_cache(rng, B, context, max_blocks)
    # values over the whole cache are as large as the new rows', so a row read before it was written shows
    qkv = dev(rng.standard_normal((steps, B, (N_Q + 2 * N_KV) * D)).astype(np.float16))
    pos = dev((context + np.arange(steps, dtype=np.int32)[:, None]).repeat(B, 1))
    return dict(kc=kc, vc=vc, bt=dev(bt), qkv=qkv, pos=pos, seq=pos + 1, freqs=dev(oracle.rope_freqs(D, 1e6)),
                w=dev(rng.uniform(0.5, 1.5, D).astype(np.float16)))


@pytest.mark.parametrize("B,context,splits", [(1, 990, 0), (1, 1000, 4), (8, 500, 0), (1, 40, 1)])
@pytest.mark.parametrize("writer", ["fused", "kvwrite", "mixed"])
def test_consecutive_positions_back_to_back(ctx, oracle, B, context, splits, writer):
    """Twenty consecutive positions of one layer with no other kernel between the calls, over a block boundary: each call reads the
    rows that the one directly ahead writes. The same bits as with a synchronisation after every call."""
    steps, max_blocks, layer, sm = 20, 128, 1, 1.0 / np.sqrt(D)
    c = chained_setup(oracle, B, context, steps, max_blocks)

    def run(sync):
        dk, dv = dev(c["kc"]), dev(c["vc"])
        out = torch.zeros((steps, B, N_Q, D), dtype=torch.float16, device="cuda")
        q = torch.zeros((steps, B, N_Q, D), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        for i in range(steps):
            if writer == "fused" or (writer == "mixed" and i % 2):
                ctx.qkv_attention_decode(c["qkv"][i], c["w"], c["w"], 1e-6, c["freqs"], c["pos"][i], dk, dv, c["bt"], c["seq"][i], out[i],
                                         B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV, context_splits=splits)
            else:
                ctx.qknorm_rope_kvwrite(c["qkv"][i], c["w"], c["w"], 1e-6, c["freqs"], c["pos"][i], c["bt"], max_blocks, dk, dv, layer,
                                        LAYERS, B, N_Q, N_KV, D, q[i])
                if writer == "mixed" or i % 3 == 2:  # (two writes ahead of one read, too)
                    ctx.paged_attention_decode(q[i], dk, dv, c["bt"], c["seq"][i], out[i], B, N_Q, D, max_blocks, sm, layer, LAYERS,
                                               N_KV, context_splits=splits)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        ctx.check_device_status()
        return out, dk, dv

    want = run(True)
    for _ in range(3):
        for w, g in zip(want, run(False)):
            assert torch.equal(w.view(torch.int16), g.view(torch.int16))


def test_prompt_written_then_read_at_once(ctx, oracle):
    """A prompt's K and V written as one batch of positions of one sequence, the attention over them the next call."""
    tokens, max_blocks, layer, sm = 900, 64, 2, 1.0 / np.sqrt(D)
    rng = np.random.default_rng(5)
    kc, vc, bt = make_cache(rng, 1, tokens, max_blocks)
    dbt, dqkv = dev(bt), dev(rng.standard_normal((tokens, (N_Q + 2 * N_KV) * D)).astype(np.float16))
    tables = dbt.expand(tokens, max_blocks).contiguous()
    pos, seq = torch.arange(tokens, dtype=torch.int32, device="cuda"), torch.full((1,), tokens, dtype=torch.int32, device="cuda")
    freqs, q = dev(oracle.rope_freqs(D, 1e6)), torch.empty((tokens, N_Q, D), dtype=torch.float16, device="cuda")
    outs = []
    for sync in (True, False, False):
        dk, dv = dev(kc), dev(vc)
        out = torch.empty((1, N_Q, D), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        ctx.qknorm_rope_kvwrite(dqkv, None, None, 1e-6, freqs, pos, tables, max_blocks, dk, dv, layer, LAYERS, tokens, N_Q, N_KV, D, q)
        if sync:
            torch.cuda.synchronize()
        ctx.paged_attention_decode(q[-1], dk, dv, dbt, seq, out, 1, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV)
        torch.cuda.synchronize()
        outs.append(out.view(torch.int16))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("B,positions,splits", [(1, [1937], 0), (8, [1024] * 8, 0), (3, [5, 300, 1000], 3)])
def test_attention_ahead_equals_the_plain_call(ctx, oracle, B, positions, splits):
    """The form that may read its inputs early, with all of them complete: the plain form's bits."""
    rng = np.random.default_rng(B)
    max_blocks, layer, sm = 128, 2, 1.0 / np.sqrt(D)
    kc, vc, bt = make_cache(rng, B, max(positions), max_blocks)
    qkv, w, fr = dev(rng.standard_normal((B, (N_Q + 2 * N_KV) * D)).astype(np.float16)), dev(rng.uniform(0.5, 1.5, D).astype(np.float16)), dev(oracle.rope_freqs(D, 1e6))
    pos, seq, dbt = dev(np.array(positions, np.int32)), dev(np.array(positions, np.int32) + 1), dev(bt)
    res = []
    for ahead in (False, True):
        dk, dv = dev(kc), dev(vc)
        out, xq, xs = torch.empty((B, N_Q, D), dtype=torch.float16, device="cuda"), torch.empty((B, N_Q * D), dtype=torch.int8, device="cuda"), torch.empty((B, N_Q * D // 64), device="cuda")
        torch.cuda.synchronize()
        ctx.qkv_attention_decode(qkv, w, w, 1e-6, fr, pos, dk, dv, dbt, seq, out, B, N_Q, D, max_blocks, sm, layer, LAYERS, N_KV,
                                 quant_group_size=64, Xq=xq, Xs=xs, context_splits=splits, ahead=ahead)
        torch.cuda.synchronize()
        res.append((out.view(torch.int16), xq, xs, dk.view(torch.int16), dv.view(torch.int16)))
    assert all(torch.equal(a, b) for a, b in zip(*res))
