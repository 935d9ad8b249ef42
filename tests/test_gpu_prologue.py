"""GPU tests of the two pre-operator kernels, bit-exact against the CPU restatement (integer and
byte work): block schedule and per-token-group fp8 quantisation, then the whole call-site sequence
of extra/sglang.patch:25-41 end to end."""
import pytest
import torch

from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,e,k,block", [(1, 257, 9, 16), (4, 8, 2, 8), (16, 8, 2, 16), (64, 257, 9, 8),
                                         (113, 257, 9, 16), (114, 257, 9, 16), (300, 37, 9, 32),
                                         (1024, 512, 10, 64), (4096, 257, 9, 128), (8192, 257, 9, 72)])
def test_moe_align_block_size_matches_oracle_exactly(m, e, k, block):
    from alpha_moe_b200.prologue import moe_align_block_size
    g = torch.Generator().manual_seed(m + e)
    ids, _ = orc.route_topk(torch.randn(m, e, generator=g), k)
    want = orc.moe_align_block_size(ids, block, e)
    got = moe_align_block_size(ids.cuda(), block, e)
    torch.cuda.synchronize()
    for a, b, name in zip(got, want, ("sorted_token_ids", "expert_ids", "num_tokens_post_padded")):
        assert torch.equal(a.cpu(), b), name


@pytest.mark.parametrize("numel", [1, 31, 32, 33, 512, 513, 1024, 1025, 1537, 2047, 2048, 2049])
@pytest.mark.parametrize("e,block", [(1, 8), (257, 16), (1023, 8), (1024, 128)])
def test_schedule_at_the_edges_of_the_single_cta_kernel(numel, e, block):
    """One CTA builds the schedule of up to 2048 assignments (16 warps of up to four rounds of 32); more, and more than
    1024 with very many slots to fill (1024 experts, blocks of 128), take the multi-CTA kernel: exact on both sides of
    every edge, with one expert and with the most there can be, for random ids and for all assignments going to the last
    expert."""
    from alpha_moe_b200.prologue import moe_align_block_size
    g = torch.Generator().manual_seed(numel + e)
    for ids in (torch.randint(0, e, (numel, 1), generator=g, dtype=torch.int32),
                torch.full((numel, 1), e - 1, dtype=torch.int32)):
        got = moe_align_block_size(ids.cuda(), block, e)
        for a, b, name in zip(got, orc.moe_align_block_size(ids, block, e),
                              ("sorted_token_ids", "expert_ids", "num_tokens_post_padded")):
            assert torch.equal(a.cpu(), b), name


@pytest.mark.parametrize("numel", [1, 33, 700, 1024, 1500, 2048])
@pytest.mark.parametrize("e", [8, 257])
def test_small_schedules_ignore_ids_out_of_range(numel, e):
    """The one-CTA schedule counts and scatters only ids in [0, E): -1, E and large ids take no slot, wherever they stand
    in a warp, and with nothing else there is no block at all."""
    from alpha_moe_b200.prologue import moe_align_block_size
    g = torch.Generator().manual_seed(numel + e)
    ids = torch.randint(0, e, (numel, 1), generator=g, dtype=torch.int32)
    bad = torch.tensor([-1, e, 1 << 30, -(1 << 31)], dtype=torch.int32)
    hit = torch.rand(numel, generator=g) < 0.3
    ids[hit, 0] = bad[torch.randint(0, 4, (int(hit.sum()),), generator=g)]
    sid, eid, npp = [t.cpu() for t in moe_align_block_size(ids.cuda(), 16, e)]
    want, blocks = [], []
    for x in range(e):
        mine = [i for i in range(numel) if int(ids[i]) == x]
        pad = -len(mine) % 16
        want += mine + [numel] * pad
        blocks += [x] * ((len(mine) + pad) // 16)
    assert int(npp) == len(want) and sid[:len(want)].tolist() == want and eid[:len(blocks)].tolist() == blocks
    assert (sid[len(want):] == numel).all()
    none = bad[torch.randint(0, 4, (numel, 1), generator=g)]
    sid, eid, npp = moe_align_block_size(none.cuda(), 16, e)
    assert int(npp) == 0 and bool((sid == numel).all())


def test_moe_align_more_chunks_than_fit_on_the_gpu_and_many_experts():
    """About a million assignments are more 1024-assignment chunks than can be resident at once, so the schedule is
    built by two launches instead of one cooperative launch; 1000 experts exercises several experts per thread in
    the offset computation.  Both bit-exact against the CPU restatement."""
    from alpha_moe_b200.prologue import moe_align_block_size
    g = torch.Generator().manual_seed(11)
    for m, e, k, block in ((130000, 257, 9, 128), (3000, 1000, 6, 16)):
        ids = torch.randint(0, e, (m, k), generator=g, dtype=torch.int32)
        want = orc.moe_align_block_size(ids, block, e)
        got = moe_align_block_size(ids.cuda(), block, e)
        torch.cuda.synchronize()
        for a, b, name in zip(got, want, ("sorted_token_ids", "expert_ids", "num_tokens_post_padded")):
            assert torch.equal(a.cpu(), b), f"{name} M={m} E={e}"


def test_moe_align_duplicates_skew_and_out_of_range_ids():
    from alpha_moe_b200.prologue import moe_align_block_size
    g = torch.Generator().manual_seed(0)
    # everything routed to two experts, duplicates inside a token (reference test generator draws with replacement)
    ids = torch.randint(0, 2, (700, 9), generator=g, dtype=torch.int32) * 5
    want = orc.moe_align_block_size(ids, 16, 8)
    got = moe_align_block_size(ids.cuda(), 16, 8)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)
    # ids outside [0, E) are ignored (they never reach a block)
    bad = ids.clone()
    bad[::7, 0] = -1
    bad[3::11, 1] = 8
    sid, eid, npp = [t.cpu() for t in moe_align_block_size(bad.cuda(), 16, 8)]
    flat = bad.reshape(-1)
    live = sid[: int(npp)]
    real = live[live < flat.numel()]
    assert sorted(real.tolist()) == [i for i in range(flat.numel()) if 0 <= int(flat[i]) < 8]


@pytest.mark.parametrize("m,k", [(1, 128), (3, 512), (64, 7168), (1000, 2048), (8192, 7168)])
def test_group_quant_matches_oracle_bit_for_bit(m, k):
    from alpha_moe_b200.prologue import per_token_group_quant_fp8
    g = torch.Generator().manual_seed(m * 7 + k)
    x = (torch.randn(m, k, generator=g) * torch.rand(m, 1, generator=g) * 3).to(torch.bfloat16)
    x[0, :128] = 0                                     # an all-zero group: scale = 1e-10 / 448
    if m > 2:
        x[2, 5] = 300.0                                # an outlier
    want_q, want_s = orc.quant_token_groups(x)
    xd = x.cuda()
    q, s = per_token_group_quant_fp8(xd)
    torch.cuda.synchronize()
    assert torch.equal(s.cpu(), want_s)
    assert torch.equal(q.cpu().view(torch.uint8), want_q.view(torch.uint8))
    assert torch.equal(xd.cpu(), x)                    # source untouched
    q2, s2 = per_token_group_quant_fp8(xd, zero_input=True)
    torch.cuda.synchronize()
    assert torch.equal(q2.cpu().view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(s2.cpu(), want_s)
    assert (xd == 0).all()


@pytest.mark.parametrize("m,e,k,hidden,block", [(1, 257, 9, 7168, 16), (7, 8, 2, 128, 8), (64, 512, 10, 2048, 16),
                                                (113, 257, 9, 7168, 32), (114, 257, 9, 7168, 16), (500, 37, 9, 1024, 64),
                                                (227, 257, 9, 7168, 16), (228, 257, 9, 1024, 16),
                                                (1100, 64, 1, 9216, 64), (1100, 64, 1, 9344, 64), (2048, 1024, 1, 128, 128)])
def test_quant_and_align_in_one_call_matches_oracle_bit_for_bit(m, e, k, hidden, block):
    """Quantisation and schedule as one launch (M * top_k <= 1024, or up to 2048 with few slots and groups) or as the two
    separate launches (the rest), on both sides of each line, against the CPU restatement of each; with and without
    clearing the source."""
    from alpha_moe_b200.prologue import quant_and_align
    g = torch.Generator().manual_seed(3 * m + e)
    x = (torch.randn(m, hidden, generator=g) * torch.rand(m, 1, generator=g) * 3).to(torch.bfloat16)
    x[0, :128] = 0
    ids, _ = orc.route_topk(torch.randn(m, e, generator=g), k)
    want_q, want_s = orc.quant_token_groups(x)
    want_sched = orc.moe_align_block_size(ids, block, e)
    for zero in (False, True):
        xd = x.cuda()
        q, s, sid, eid, npp = quant_and_align(xd, ids.cuda(), block, e, zero_input=zero)
        torch.cuda.synchronize()
        assert torch.equal(q.cpu().view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(s.cpu(), want_s)
        for a, b, name in zip((sid, eid, npp), want_sched, ("sorted_token_ids", "expert_ids", "num_tokens_post_padded")):
            assert torch.equal(a.cpu(), b), name
        assert (xd == 0).all() if zero else torch.equal(xd.cpu(), x)


def test_call_site_sequence_end_to_end():
    """quantise -> zero the activations -> schedule -> fused operator accumulating into the activation
    buffer, exactly the sequence of the reference's call site (extra/sglang.patch:30-41)."""
    import alpha_moe  # noqa: F401
    from alpha_moe_b200.prologue import moe_align_block_size, sglang_per_token_group_quant_fp8
    e, k, inter, m, top_k = 16, 1024, 256, 50, 4
    g = torch.Generator().manual_seed(3)
    w, w_scale, w2, w2_scale = orc.make_weights(e, k, inter, g)
    hidden = torch.randn(m, k, generator=g).to(torch.bfloat16)
    ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
    xq, xs = orc.quant_token_groups(hidden)
    sid, eid, npp = orc.moe_align_block_size(ids, 16, e)
    ref = orc.fused_moe_w8a8_up_down_oracle(xq, xs, w, w_scale, w2, w2_scale, sid, eid, npp, wts, top_k, 16, 2.5)

    hs = hidden.cuda()
    a, a_scale = sglang_per_token_group_quant_fp8(hs, 128, zero_input=True)
    s_ids, e_ids, n_pad = moe_align_block_size(ids.cuda(), 16, e)
    torch.ops.alpha_moe.fused_moe_w8a8_up_down(a, a_scale, w.cuda(), w_scale.cuda(), w2.cuda(), w2_scale.cuda(),
                                               s_ids, e_ids, n_pad, wts.cuda(), hs, top_k, 16, 32, 8, 3, 2.5)
    torch.cuda.synchronize()
    assert orc.rel_l2(hs.cpu(), ref) <= 2e-2


@pytest.mark.parametrize("m,conf", [(50, {"block_m": 16, "block_n": 32, "warp_n": 8, "stages": 3}),
                                     (300, {"block_m": 128, "block_n": 64, "warp_n": 4, "stages": 3})])
def test_fused_experts_single_call_matches_the_step_by_step_sequence(m, conf, tmp_path):
    """alpha_moe_b200.layer.fused_experts_impl (one C-ABI call for the body of the reference's patched
    fused_experts_impl, extra/sglang.patch:25-40) against the oracle, with the knobs given directly and
    through a table file + ALPHA_MOE_CONFIG-style look-up."""
    import json
    from alpha_moe_b200.layer import fused_experts_impl
    e, k, inter, top_k = 16, 1024, 256, 4
    g = torch.Generator().manual_seed(5 + m)
    w, w_scale, w2, w2_scale = orc.make_weights(e, k, inter, g)
    hidden = torch.randn(m, k, generator=g).to(torch.bfloat16)
    ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
    xq, xs = orc.quant_token_groups(hidden)
    bm = conf["block_m"]
    sid, eid, npp = orc.moe_align_block_size(ids, bm, e)
    ref = orc.fused_moe_w8a8_up_down_oracle(xq, xs, w, w_scale, w2, w2_scale, sid, eid, npp, wts, top_k, bm, 2.5)
    dw = [t.cuda() for t in (w, w_scale, w2, w2_scale)]

    hs = hidden.cuda()
    out = fused_experts_impl(hs, *dw, wts.cuda(), ids.cuda(), routed_scaling_factor=2.5, config=conf)
    torch.cuda.synchronize()
    assert out.data_ptr() == hs.data_ptr()            # result in place, as at the reference's call site
    assert orc.rel_l2(hs.cpu(), ref) <= 2e-2

    table = tmp_path / "moe.json"
    table.write_text(json.dumps({str(m): conf}))
    hs2 = hidden.cuda()
    fused_experts_impl(hs2, *dw, wts.cuda(), ids.cuda(), routed_scaling_factor=2.5, config=str(table))
    torch.cuda.synchronize()
    assert torch.equal(hs2.cpu(), hs.cpu()) or orc.rel_l2(hs2.cpu(), hs.cpu()) <= 1e-2   # reduction order may differ


def test_back_to_back_layers_with_changing_inputs_eager_and_from_a_graph():
    """The operator is launched with programmatic stream serialisation (its CTAs may be scheduled while the
    quantise/schedule kernel in front of it is still running, and wait for that kernel's completion before reading
    anything).  Several layers in a row, each with its own activations and routing but through the same scratch
    memory, must each see their own schedule and activations - eagerly and replayed from one CUDA graph."""
    from alpha_moe_b200.layer import fused_experts_impl
    e, k, inter, top_k = 16, 1024, 256, 4
    g = torch.Generator().manual_seed(77)
    w, w_scale, w2, w2_scale = orc.make_weights(e, k, inter, g)
    dw = [t.cuda() for t in (w, w_scale, w2, w2_scale)]
    steps = []
    for m, bm, bn, wn in ((3, 16, 32, 8), (50, 16, 32, 8), (50, 32, 64, 4), (200, 128, 64, 4), (7, 8, 32, 8)):
        hidden = torch.randn(m, k, generator=g).to(torch.bfloat16)
        ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
        xq, xs = orc.quant_token_groups(hidden)
        sid, eid, npp = orc.moe_align_block_size(ids, bm, e)
        ref = orc.fused_moe_w8a8_up_down_oracle(xq, xs, w, w_scale, w2, w2_scale, sid, eid, npp, wts, top_k, bm, 2.5)
        conf = {"block_m": bm, "block_n": bn, "warp_n": wn, "stages": 3}
        steps.append((hidden, ids.cuda(), wts.cuda(), conf, ref))

    def run_all(bufs):
        for (hidden, ids, wts, conf, _), hs in zip(steps, bufs):
            fused_experts_impl(hs, *dw, wts, ids, routed_scaling_factor=2.5, config=conf)

    bufs = [s[0].cuda() for s in steps]
    run_all(bufs)
    torch.cuda.synchronize()
    for (_, _, _, conf, ref), hs in zip(steps, bufs):
        assert orc.rel_l2(hs.cpu(), ref) <= 2e-2, conf

    static = [s[0].cuda() for s in steps]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run_all([b.clone() for b in static])              # warm-up on the capture stream
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run_all(static)
    for rep in range(2):
        for (hidden, _, _, _, _), hs in zip(steps, static):
            hs.copy_(hidden.cuda())
        graph.replay()
        torch.cuda.synchronize()
        for (_, _, _, conf, ref), hs in zip(steps, static):
            assert orc.rel_l2(hs.cpu(), ref) <= 2e-2, (rep, conf)
    from alpha_moe_b200 import capi
    assert capi.read_status(reset=True)[0] == 0


@pytest.mark.parametrize("m,top_k,e,k,inter,bm,stages", [
    (1, 1, 1, 128, 128, 16, 1),            # one assignment, one chunk, a ring of one slot
    (1, 9, 24, 7168, 256, 16, 4),          # one token at the DeepSeek-V3 TP8 shard's sizes
    (5, 9, 257, 1024, 256, 16, 2),
    (3, 10, 512, 2048, 256, 16, 4),
    (14, 9, 40, 384, 384, 8, 3),           # several blocks of an expert, three slices
    (28, 9, 257, 512, 256, 8, 5),          # two slices per CTA (block_n = 64 from here on where even)
    (57, 9, 257, 256, 512, 16, 3),         # 513 assignments: the third of a thread's eight
    (256, 8, 1024, 256, 256, 8, 5),        # 2048 assignments, the last that a thread reads once; 1024 experts
    (205, 10, 33, 128, 256, 16, 2),        # 2050: ids read twice
    (205, 10, 300, 128, 256, 32, 2),       # tiles of 32 and 64 tokens
    (33, 9, 1024, 256, 512, 64, 2),
    (819, 10, 50, 128, 256, 48, 2),        # 8190 assignments, the last of a thread's 32
    (819, 10, 50, 128, 256, 32, 2),        # the same in tiles of 32
    (820, 10, 50, 128, 256, 64, 2),        # 8200: the schedule kernel again
])
@pytest.mark.parametrize("routing", ["topk", "duplicates", "outside", "none"])
def test_small_batches_whose_operator_makes_its_own_schedule(m, top_k, e, k, inter, bm, stages, routing):
    """Up to 8192 assignments in blocks of up to 64 the layer call launches no schedule kernel: every CTA derives its block from
    the routing.  Token by token against the oracle on the reference's schedule and against the steps one by one, with experts
    chosen twice by a token, ids outside [0, E) (ignored) and no valid id at all; eagerly and from a graph."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.layer import fused_experts_impl
    g = torch.Generator().manual_seed(100 * m + top_k)
    w, w_scale, w2, w2_scale = orc.make_weights(min(e, 24), k, inter, g)
    if e > 24:                                             # few distinct experts, at both ends and in the middle of the range
        pick = torch.arange(e) % 24
        w, w2 = (t.view(torch.uint8)[pick].view(torch.float8_e4m3fn) for t in (w, w2))
        w_scale, w2_scale = w_scale[pick], w2_scale[pick]
    # every expert has a size of its own, and every other 24 the other sign: no expert passes for another with the same weights
    size = (0.5 + 1.5 * torch.rand(e, generator=g)) * (1 - 2 * (torch.arange(e) // 24 % 2))
    w2_scale = w2_scale * size[:, None, None]
    hidden = torch.randn(m, k, generator=g).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(e, generator=g)[:top_k] for _ in range(m)]).to(torch.int32)
    if routing == "duplicates":
        ids = torch.randint(max(0, e - 3), e, (m, top_k), generator=g, dtype=torch.int32)
    elif routing == "outside":
        ids[::2, ::2] = -1
        ids[1::2, ::3] = e
    elif routing == "none":
        ids[:] = -7
    wts = 0.5 + torch.rand(m, top_k, generator=g)
    valid = (ids >= 0) & (ids < e)
    xq, xs = orc.quant_token_groups(hidden)
    sid, eid, npp = orc.moe_align_block_size(ids.clamp(0, e - 1), bm, e)      # (an ignored id is one of weight 0)
    ref = orc.fused_moe_w8a8_up_down_oracle(xq, xs, w, w_scale, w2, w2_scale, sid, eid, npp, wts * valid, top_k, bm, 2.5)
    args = [t.cuda() for t in (w, w_scale, w2, w2_scale, wts, ids)]
    conf = {"block_m": bm, "block_n": 32 if m < 28 else 64, "warp_n": 8 if m < 28 else 4, "stages": stages}

    def call(hs):
        return fused_experts_impl(hs, *args, routed_scaling_factor=2.5, config=conf)

    def token_error(got, want):
        return float(((got.float() - want.float()).norm(dim=1) / want.float().norm(dim=1).clamp_min(1e-30))[valid.any(1)].max())

    from alpha_moe_b200.prologue import moe_align_block_size, per_token_group_quant_fp8
    steps = torch.zeros(m, k, dtype=torch.bfloat16, device="cuda")
    torch.ops.alpha_moe.fused_moe_w8a8_up_down(*per_token_group_quant_fp8(hidden.cuda()), *args[:4],
                                               *moe_align_block_size(args[5], bm, e), args[4], steps, top_k, *conf.values(), 2.5)
    hs = hidden.cuda()
    call(hs)
    static = hidden.cuda()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(static)
    for got in (hs, static):
        if got is static:
            graph.replay()
        torch.cuda.synchronize()
        assert capi.read_status(reset=True)[0] == 0
        assert not got[~valid.any(1)].any()
        if valid.any():
            # A token's sum takes top_k x slice groups bf16 additions, each off by up to 2^-9 of a partial sum, at random: at most
            # sqrt(30) x 2^-9 = 1.1 %, and its fp8 intermediates may round to the neighbour here and there.  A lost, doubled or
            # misplaced assignment is at least 0.5 x 0.5 of a sum of ten that are 1.5 x 2 at most, in quadrature: 2.6 %.
            assert token_error(got.cpu(), ref) <= 2.5e-2
            assert token_error(got.cpu(), steps.cpu()) <= 2.5e-2


@pytest.mark.parametrize("m,k,inter,bm,bn,stages", [(1, 7168, 256, 16, 32, 4), (5, 1024, 256, 16, 32, 2), (24, 256, 512, 8, 64, 5),
                                                    (203, 256, 256, 16, 64, 2), (500, 256, 256, 32, 64, 2)])
def test_routing_written_right_in_front_of_the_call(m, k, inter, bm, bn, stages):
    """The operator that makes its own schedule reads the routing before it waits for the quantiser.  A kernel directly in front of
    the call writes activations, ids and weights, with other values at every replay of one graph and in eager calls in a row."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.layer import fused_experts_impl
    from alpha_moe_b200.prologue import moe_align_block_size, per_token_group_quant_fp8
    e, top_k, sets = 64, 9, 8
    g = torch.Generator(device="cuda").manual_seed(m)
    w = torch.randn(e, 2 * inter, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    w2 = torch.randn(e, k, inter, generator=g, device="cuda").to(torch.float8_e4m3fn)
    ws = torch.full((e, inter // 64, k // 128), 0.02, device="cuda")
    w2s = torch.rand(e, k // 128, inter // 128, generator=g, device="cuda") * 0.02 + 0.01
    x_all = torch.randn(sets, m, k, generator=g, device="cuda").to(torch.bfloat16)
    ids_all = torch.randint(0, e, (sets, m, top_k), generator=g, device="cuda", dtype=torch.int32)
    wts_all = torch.rand(sets, m, top_k, generator=g, device="cuda") + 0.5
    conf = dict(block_m=bm, block_n=bn, warp_n=256 // bn, stages=stages)
    want = []
    for x, ids, wts in zip(x_all, ids_all, wts_all):
        out = torch.zeros_like(x)
        torch.ops.alpha_moe.fused_moe_w8a8_up_down(*per_token_group_quant_fp8(x), w, ws, w2, w2s, *moe_align_block_size(ids, bm, e),
                                                   wts, out, top_k, *conf.values(), 1.0)
        want.append(out)
    torch.cuda.synchronize()
    turn = torch.zeros(1, dtype=torch.int64, device="cuda")
    hs, wts, ids = x_all[0].clone(), wts_all[0].clone(), ids_all[0].clone()

    def write_and_call():
        torch.index_select(x_all, 0, turn, out=hs.unsqueeze(0))
        torch.index_select(wts_all, 0, turn, out=wts.unsqueeze(0))
        torch.index_select(ids_all, 0, turn, out=ids.unsqueeze(0))
        fused_experts_impl(hs, w, ws, w2, w2s, wts, ids, config=conf)
        turn.add_(1)

    write_and_call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        write_and_call()
    for step in (graph.replay, write_and_call):
        turn.zero_()
        got = []
        for _ in range(sets):
            step()
            got.append(hs.clone())
        torch.cuda.synchronize()
        assert capi.read_status(reset=True)[0] == 0
        for a, b in zip(got, want):
            assert float(((a.float() - b.float()).norm(dim=1) / b.float().norm(dim=1)).max()) <= 2.5e-2      # (bound as above)


@pytest.mark.parametrize("ks", [1, 2, 3, 4, 5, 6, 7, 8])
def test_own_schedule_in_clusters_of_every_size(ks):
    """Both exchanges of the partial sums - few live columns, sent; more, read from the peers - with the blocks taken from the back."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.layer import fused_experts_impl
    e, k, inter, top_k = 16, 1152, 256, 4
    g = torch.Generator().manual_seed(ks)
    w, w_scale, w2, w2_scale = orc.make_weights(e, k, inter, g)
    dw = [t.cuda() for t in (w, w_scale, w2, w2_scale)]
    capi.set_ksplit(ks)
    try:
        for m, spread in ((1, e), (3, e), (12, 5), (40, e)):        # tokens, experts they choose from: 1 to 16 live columns
            hidden = torch.randn(m, k, generator=g).to(torch.bfloat16)
            ids = torch.stack([torch.randperm(spread, generator=g)[:top_k] for _ in range(m)]).to(torch.int32)
            wts = 0.5 + torch.rand(m, top_k, generator=g)
            sid, eid, npp = orc.moe_align_block_size(ids, 16, e)
            ref = orc.fused_moe_w8a8_up_down_oracle(*orc.quant_token_groups(hidden), w, w_scale, w2, w2_scale, sid, eid, npp, wts,
                                                    top_k, 16, 1.0)
            hs = hidden.cuda()
            fused_experts_impl(hs, *dw, wts.cuda(), ids.cuda(), config=dict(block_m=16, block_n=32, warp_n=8, stages=3))
            torch.cuda.synchronize()
            assert capi.read_status(reset=True)[0] == 0
            err = (hs.cpu().float() - ref.float()).norm(dim=1) / ref.float().norm(dim=1)
            assert float(err.max()) <= 2.5e-2, (m, spread)
    finally:
        capi.set_ksplit(0)


@pytest.mark.parametrize("m,top_k,e,inter,bm,bn,stages", [
    (1, 1, 1, 256, 16, 32, 1),             # one block and no slot behind it that an expert leaves empty
    (1, 9, 257, 256, 16, 32, 4),           # clusters, whose blocks go from the back
    (5, 9, 257, 256, 16, 32, 2),
    (28, 9, 1024, 512, 8, 64, 5),          # most of the schedule lies behind the last block
    (114, 9, 33, 256, 16, 32, 3),          # 1026 assignments; no clusters
    (205, 10, 300, 512, 32, 64, 2),
    (819, 10, 50, 512, 48, 64, 2),
    (819, 10, 50, 512, 128, 64, 3),        # the schedule kernel
])
@pytest.mark.parametrize("routing", ["topk", "outside", "none"])
def test_single_call_leaves_the_schedule_in_the_callers_buffers(m, top_k, e, inter, bm, bn, stages, routing):
    """The C entry's schedule buffers hold the schedule kernel's words afterwards, whichever form the operator took."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.prologue import moe_align_block_size, per_token_group_quant_fp8
    k = 256
    g = torch.Generator().manual_seed(m + e)
    ids = torch.stack([torch.randperm(e, generator=g)[:top_k] for _ in range(m)]).to(torch.int32)
    if routing == "outside":
        ids[::2, ::2] = -1
        ids[1::2, ::3] = e
    elif routing == "none":
        ids[:] = e + 3
    ids, hidden = ids.cuda(), torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    want = (*moe_align_block_size(ids, bm, e), *per_token_group_quant_fp8(hidden))
    got = [torch.full_like(t.view(torch.int32), -99) for t in want[:3]] + [torch.zeros_like(t) for t in want[3:]]
    w = torch.zeros(e, 2 * inter, k, dtype=torch.float8_e4m3fn, device="cuda")
    w2 = torch.zeros(e, k, inter, dtype=torch.float8_e4m3fn, device="cuda")
    ws, w2s = torch.ones(e, inter // 64, k // 128, device="cuda"), torch.ones(e, k // 128, inter // 128, device="cuda")
    wts = torch.ones(m, top_k, device="cuda")
    scratch = torch.empty(max(capi.align_workspace_bytes(m * top_k, e), 4), dtype=torch.uint8, device="cuda")
    capi.fused_experts(hidden.data_ptr(), got[3].data_ptr(), got[4].data_ptr(), w.data_ptr(), ws.data_ptr(), w2.data_ptr(),
                       w2s.data_ptr(), ids.data_ptr(), wts.data_ptr(), top_k, m, k, 2 * inter, e,
                       got[0].data_ptr(), got[1].data_ptr(), got[2].data_ptr(), scratch.data_ptr(), bm, bn, 256 // bn, stages,
                       1.0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert capi.read_status(reset=True)[0] == 0
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


def test_layer_call_refuses_cuda_tensors_in_the_words_of_the_host_checks():
    """fused_experts_impl checks CUDA tensors inside its operator: what _check_layer_arguments refuses is refused with the same
    message, an ABI error keeps its type, and the buffer is left alone."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.layer import _check_layer_arguments, fused_experts_impl
    e, n, k, m, top_k = 4, 256, 256, 3, 2
    f8 = torch.float8_e4m3fn
    good = dict(
        hidden_states=torch.ones(m, k, dtype=torch.bfloat16, device="cuda", requires_grad=True),
        w1=torch.zeros(e, n, k, dtype=f8, device="cuda"), w1_scale=torch.zeros(e, n // 128, k // 128, device="cuda"),
        w2=torch.zeros(e, k, n // 2, dtype=f8, device="cuda"), w2_scale=torch.zeros(e, k // 128, n // 256, device="cuda"),
        topk_weights=torch.zeros(m, top_k, device="cuda"), topk_ids=torch.zeros(m, top_k, dtype=torch.int32, device="cuda"))
    conf = dict(block_m=16, block_n=32, warp_n=8, stages=3)

    def call(knobs=conf, **change):
        a = dict(good, **change)
        return fused_experts_impl(a["hidden_states"], a["w1"], a["w1_scale"], a["w2"], a["w2_scale"], a["topk_weights"],
                                  a["topk_ids"], config=knobs)

    bad = [
        dict(hidden_states=torch.zeros(m, k, device="cuda")),
        dict(hidden_states=torch.zeros(m, 2 * k, dtype=torch.bfloat16, device="cuda")[:, ::2]),
        dict(hidden_states=torch.zeros(0, k, dtype=torch.bfloat16, device="cuda")),
        dict(w1=torch.zeros(e, n, k // 2, dtype=f8, device="cuda")),
        dict(w1=torch.zeros(e, 2 * n, k, dtype=f8, device="cuda")[:, ::2]),
        dict(w2=torch.zeros(e, k, n, dtype=f8, device="cuda")),
        dict(w2=torch.zeros(e, k, n // 2, dtype=torch.uint8, device="cuda")),
        dict(w1_scale=torch.zeros(e, n // 128, k // 128 + 1, device="cuda")),
        dict(w2_scale=torch.zeros(e, k // 128, n // 256, dtype=torch.float64, device="cuda")),
        dict(w2_scale=torch.zeros(e, k // 128, n // 256)),
        dict(topk_ids=torch.zeros(m + 1, top_k, dtype=torch.int32, device="cuda")),
        dict(topk_weights=torch.zeros(m, top_k + 1, device="cuda")),
    ]
    for change in bad:
        with pytest.raises(RuntimeError) as want:
            _check_layer_arguments(**dict(good, **change))
        with pytest.raises(RuntimeError) as got:
            call(**change)
        assert str(want.value) in str(got.value), (change, str(got.value))
    for knobs in (dict(conf, block_m=0), dict(conf, stages=9), dict(conf, block_m=136)):
        with pytest.raises(RuntimeError):
            call(knobs)
    with pytest.raises(capi.AlphaMoeError, match="stages"):
        call(dict(conf, stages=9, block_m=128, block_n=64, warp_n=4))
    for block_m in (-8, 0, 12, 136):
        with pytest.raises(capi.AlphaMoeError, match="bad block_m"):
            call(dict(conf, block_m=block_m))
    assert bool((good["hidden_states"] == 1).all())
    # other dtypes and layouts of the routing are converted; a buffer that requires gradients is overwritten all the same
    out = call(topk_ids=torch.zeros(top_k, m, dtype=torch.int64, device="cuda").t(),
               topk_weights=torch.zeros(m, top_k, dtype=torch.float64, device="cuda"))
    assert out is good["hidden_states"] and not out.detach().any() and out.grad_fn is None


def test_layer_call_on_the_c_library_alone_matches_the_operator(monkeypatch):
    """Without the torch operator's library the layer call makes its checks and buffers in Python; also on another stream, with
    routing that has to be converted, and with the error type of the C ABI."""
    from alpha_moe_b200 import capi, layer
    e, k, inter, m, top_k = 8, 256, 256, 130, 8            # 1040 assignments: a workspace, too
    g = torch.Generator().manual_seed(3)
    dw = [t.cuda() for t in orc.make_weights(e, k, inter, g)]
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
    ids, wts = ids.long().cuda(), wts.double().cuda()
    conf = dict(block_m=16, block_n=32, warp_n=8, stages=3)
    want = layer.fused_experts_impl(x.clone(), *dw, wts, ids, config=conf)
    monkeypatch.setattr(layer, "_fused_experts", layer._through_c_abi)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = layer.fused_experts_impl(x.clone(), *dw, wts, ids, config=conf)
    torch.cuda.synchronize()
    assert orc.rel_l2(got.cpu(), want.cpu()) <= 1e-2
    with pytest.raises(capi.AlphaMoeError, match="stages"):
        layer.fused_experts_impl(x.clone(), *dw, wts, ids, config=dict(conf, stages=9))
    with pytest.raises(RuntimeError, match="w1_scale"):
        layer.fused_experts_impl(x.clone(), dw[0], dw[1][:, 1:], *dw[2:], wts, ids, config=conf)


@pytest.mark.parametrize("backend", ["eager", "aot_eager"])
def test_layer_call_inside_a_compiled_function(backend):
    """torch.compile breaks its graph at the layer call, as it did when the call went through ctypes."""
    from alpha_moe_b200.layer import fused_experts_impl
    e, k, inter, m, top_k = 8, 256, 256, 5, 2
    g = torch.Generator().manual_seed(9)
    dw = [t.cuda() for t in orc.make_weights(e, k, inter, g)]
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
    ids, wts = ids.cuda(), wts.cuda()
    conf = dict(block_m=16, block_n=32, warp_n=8, stages=3)

    def layer(h):
        return fused_experts_impl(h, *dw, wts, ids, routed_scaling_factor=2.5, config=conf) * 2

    want = layer(x.clone())
    torch._dynamo.reset()
    h = x.clone()
    got = torch.compile(layer, backend=backend)(h)
    assert orc.rel_l2(got.cpu(), want.cpu()) <= 1e-2 and orc.rel_l2(2 * h.cpu(), want.cpu()) <= 1e-2


def test_layer_call_inside_a_traced_function():
    """torch.jit.trace records the layer call: the trace computes the layer on other activations and another routing."""
    from alpha_moe_b200.layer import fused_experts_impl
    e, k, inter, m, top_k = 8, 256, 256, 5, 2
    g = torch.Generator().manual_seed(11)
    dw = [t.cuda() for t in orc.make_weights(e, k, inter, g)]
    conf = dict(block_m=16, block_n=32, warp_n=8, stages=3)

    def layer(h, wts, ids):
        return fused_experts_impl(h, *dw, wts, ids, routed_scaling_factor=2.5, config=conf) * 2

    def inputs():
        ids, wts = orc.route_topk(torch.randn(m, e, generator=g), top_k)
        return torch.randn(m, k, generator=g).to(torch.bfloat16).cuda(), wts.cuda(), ids.cuda()

    traced = torch.jit.trace(layer, inputs(), check_trace=False)
    h, wts, ids = inputs()
    want = layer(h.clone(), wts, ids)
    assert orc.rel_l2(traced(h, wts, ids).cpu(), want.cpu()) <= 1e-2


@pytest.mark.parametrize("m,top_k,e,inter,bm,bn,stages,own", [
    (1, 1, 1, 256, 16, 32, 1, True),
    (97, 9, 257, 2048, 16, 64, 2, True),         # eight slice groups: 2368 CTAs, the line on 148 SMs
    (98, 9, 257, 2048, 16, 64, 2, False),
    (1024, 8, 2, 256, 32, 64, 2, True),          # 8192 assignments
    (1025, 8, 2, 256, 32, 64, 2, False),
    (33, 9, 40, 256, 32, 32, 2, False),          # a tile of 32 with one slice, one with a ring of one slot
    (33, 9, 40, 256, 32, 64, 1, False),
    (33, 9, 40, 256, 40, 64, 2, True),           # a tile of 64 with the short ring, with a longer one
    (33, 9, 40, 256, 40, 64, 3, False),
    (33, 9, 871, 128, 16, 32, 3, False),         # more experts than the histogram has room for
])
def test_which_layer_calls_make_their_own_schedule(m, top_k, e, inter, bm, bn, stages, own, tmp_path):
    """Both sides of every line between the operator that makes its own schedule and the schedule kernel, each against the steps
    one by one, token by token."""
    from alpha_moe_b200 import capi
    from alpha_moe_b200.layer import fused_experts_impl
    from alpha_moe_b200.prologue import moe_align_block_size, per_token_group_quant_fp8
    k = 128
    g = torch.Generator(device="cuda").manual_seed(m + e)
    w = torch.randn(e, 2 * inter, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    w2 = torch.randn(e, k, inter, generator=g, device="cuda").to(torch.float8_e4m3fn)
    ws = torch.rand(e, inter // 64, 1, generator=g, device="cuda") * 0.02 + 0.01
    w2s = torch.rand(e, 1, inter // 128, generator=g, device="cuda") * 0.02 + 0.01
    ids = torch.randint(0, e, (m, top_k), generator=g, device="cuda", dtype=torch.int32)
    wts = torch.rand(m, top_k, generator=g, device="cuda") + 0.1
    hidden = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    conf = {"block_m": bm, "block_n": bn, "warp_n": 256 // bn, "stages": stages}
    xq, xs = per_token_group_quant_fp8(hidden)
    sid, eid, npp = moe_align_block_size(ids, bm, e)
    want = torch.zeros_like(hidden)
    torch.ops.alpha_moe.fused_moe_w8a8_up_down(xq, xs, w, ws, w2, w2s, sid, eid, npp, wts, want, top_k, bm, bn, 256 // bn, stages, 1.0)
    got = hidden.clone()
    fused_experts_impl(got, w, ws, w2, w2s, wts, ids, config=conf)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        fused_experts_impl(hidden, w, ws, w2, w2s, wts, ids, config=conf)
    graph.debug_dump(str(tmp_path / "graph.dot"))         # the launches' names
    names = (tmp_path / "graph.dot").read_text()
    assert "fused_moe" in names and ("group_quant" in names or "quant_and_align" in names)
    assert ("align" in names) != own
    assert capi.read_status(reset=True)[0] == 0
    err = (got.float() - want.float()).norm(dim=1) / want.float().norm(dim=1)
    assert float(err.max()) <= 2e-2
