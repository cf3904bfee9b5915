"""The kernels and dispatch rules of decode-sized calls at the sizes where they can go wrong, against the oracle: the plan
and quantisation in one launch (up to 1024 slots) and the two-pass plan beyond, split-K post passes (up to 64 rows), the
block-scale tiles that read back 8, 16 or 32 token columns, always-on experts written by the router, caller-routed batches,
and the router's candidate bounds."""

import pytest
import torch

import oracle
from helpers import BF16, check_against_oracle, make_inputs, run_cuda_forward, run_oracle_forward, to_cuda
from test_block_gpu import make_block_inputs

pytestmark = pytest.mark.gpu


# rows T*K of 1, 8, 16, 17, 64, 65, 1024 and 1025; ragged D and H; all experts selected; more experts than rows
@pytest.mark.parametrize("T,D,E,K,H", [(1, 256, 4, 1, 64), (1, 272, 8, 8, 144), (2, 1040, 16, 8, 320), (17, 256, 4, 1, 128),
                                       (8, 512, 8, 8, 1408), (13, 256, 16, 5, 208), (3, 2048, 66, 8, 1408),
                                       (1024, 128, 16, 1, 64), (1025, 144, 16, 1, 64), (128, 400, 256, 8, 48)])
def test_per_tensor_forward_at_the_edges_of_the_dispatch(T, D, E, K, H):
    inp = make_inputs(T, D, E, K, H, seed=T * 7 + K)
    out, views = run_cuda_forward(inp)
    ref, inter = run_oracle_forward(inp)
    check_against_oracle(inp, out, views, ref, inter)


# the kernel for up to 8 rows per expert on average: one token over few and many tiles, an odd number of K blocks, a single
# expert, ragged D and H, several row tiles per expert; 1024 and 1025 slots
@pytest.mark.parametrize("T,D,E,K,H", [(1, 1024, 16, 8, 128), (1, 1024, 16, 8, 640), (1, 2048, 128, 8, 768), (1, 640, 8, 3, 384),
                                       (2, 512, 8, 4, 256), (8, 512, 1, 1, 256), (9, 1024, 2, 1, 256), (24, 384, 8, 2, 576),
                                       (40, 512, 16, 3, 208), (70, 256, 32, 2, 144), (1024, 128, 256, 1, 128), (1025, 272, 160, 1, 128)])
def test_block_forward_at_the_edges_of_the_dispatch(T, D, E, K, H):
    import blackwell_moe_b200 as bw
    inp = make_block_inputs(T, D, E, K, H, seed=T + D)
    c = to_cuda(inp)
    call = lambda: bw.fp8_moe_forward(c["x"], c["w_gate"], c["q_gate"], c["q_up"], c["q_down"],
                                      c["inv_gate"], c["inv_up"], c["inv_down"], top_k=K)
    out = call()
    v = {k: t.cpu() for k, t in bw.moe_stage_views("cuda:0", T, D, H, E, K, block=True).items()}
    inter = {}
    ref = oracle.moe_forward_block_recipe(inp["x"], inp["w_gate"], inp["q_gate"], inp["q_up"], inp["q_down"],
                                          inp["inv_gate"], inp["inv_up"], inp["inv_down"], top_k=K, intermediates=inter)
    assert int(v["status"][0]) == 0
    for name, want in (("indices", "indices"), ("offsets", "offsets"), ("x_inv", "x_inv")):
        assert torch.equal(v[name], inter[want]), name
    assert torch.equal(v["row_slot"].long(), inter["sort_perm"])
    assert torch.equal(v["xq"].view(torch.uint8), inter["xq"].view(torch.uint8))
    assert (v["hq"].view(torch.uint8) != inter["hq"].view(torch.uint8)).float().mean().item() < 0.02
    assert oracle.rel_l1(v["y"], inter["y_perm"]) < 1e-2
    assert oracle.rel_l1(out.cpu(), ref) < 1e-2
    assert torch.equal(call(), out)                     # sums in a fixed order


def _rows_per_expert(counts):
    """Caller-routed batch of one slot per token in which expert e gets counts[e] rows, in no order."""
    g = torch.Generator().manual_seed(sum(counts))
    ids = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    ids = ids[torch.randperm(len(ids), generator=g)].to(torch.int32)[:, None]
    return torch.rand(len(ids), 1, generator=g) + 0.5, ids


# rows of the first expert: both sides of the 8, 16 and 32 columns that a tile reads back and holds, and of two tiles
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("D,H", [(512, 256), (400, 208)])
def test_block_tiles_at_the_edges_of_what_they_read_back(rows, D, H):
    _check_block_routed([rows, 0, 3] + [0] * 13, D, H)


# 8 rows per expert on average are the last for the small kernel: 64 and 65 rows of 8 experts
@pytest.mark.parametrize("counts", [[8] * 8, [8] * 7 + [9], [40, 0, 3, 9, 1, 11, 0, 0], [40, 0, 3, 9, 1, 11, 1, 0]])
def test_block_kernels_on_both_sides_of_eight_rows_per_expert(counts):
    _check_block_routed(counts, 384, 272)


def _check_block_routed(counts, D, H):
    import blackwell_moe_b200 as bw
    wt, ids = _rows_per_expert(counts)
    T, E = len(ids), len(counts)
    inp = make_block_inputs(T, D, E, 1, H, seed=T + D)
    c = to_cuda(inp)
    out = bw.fp8_moe_forward_routed(c["x"], wt.cuda(), ids.cuda(), c["q_gate"], c["q_up"], c["q_down"],
                                    c["inv_gate"], c["inv_up"], c["inv_down"])
    v = {k: t.cpu() for k, t in bw.moe_stage_views("cuda:0", T, D, H, E, 1, block=True).items()}
    inter = {}
    ref = oracle.moe_forward_block_recipe(inp["x"], None, inp["q_gate"], inp["q_up"], inp["q_down"], inp["inv_gate"],
                                          inp["inv_up"], inp["inv_down"], routing=(wt, ids), intermediates=inter)
    assert int(v["status"][0]) == 0
    assert torch.equal(v["offsets"], inter["offsets"]) and torch.equal(v["x_inv"], inter["x_inv"])
    assert (v["hq"].view(torch.uint8) != inter["hq"].view(torch.uint8)).float().mean().item() < 0.02
    assert max(oracle.rel_l1(v["y"][i], inter["y_perm"][i]) for i in range(T)) < 2e-2
    assert oracle.rel_l1(out.cpu(), ref) < 1e-2


# 8, 64, 72 and 1200 rows: fused and separate requantisation; both forms of the combine (rows of 512 and 272 columns)
@pytest.mark.parametrize("T,D", [(1, 512), (8, 512), (9, 512), (150, 512), (9, 272), (150, 272)])
def test_always_on_experts_share_one_scale_and_follow_the_routed_slots(T, D):
    import blackwell_moe_b200 as bw
    E, K, H, S = 16, 6, 256, 2
    inp = make_inputs(T, D, E, K, H, seed=T + 3)
    shared = [oracle.quant_fp8_e4m3((torch.randn(a, b, generator=torch.Generator().manual_seed(i)) * 0.02).to(BF16))
              for i, (a, b) in enumerate(((D, S * H), (D, S * H), (S * H, D)))]
    c = to_cuda(inp)
    stacked = bw.stack_shared_experts(c["q_gate"], c["q_up"], c["q_down"], c["s_gate"], c["s_up"], c["s_down"],
                                      *[q.cuda() for q, _ in shared], *[s.float().cuda() for _, s in shared])
    out = bw.fp8_moe_forward_shared(c["x"], c["w_gate"], *stacked[:6], top_k=K, n_shared=S, routed_scale=1.5)
    routed, _ = run_oracle_forward(inp)
    sh = oracle.shared_expert_fp8(inp["x"], *[q for q, _ in shared], *[s for _, s in shared])
    ref = ((routed * 1.5).to(BF16) + sh).to(BF16)
    assert oracle.rel_l1(out.cpu(), ref) < 1e-2


@pytest.mark.parametrize("block", [False, True])
@pytest.mark.parametrize("T", [1, 37, 700])
def test_caller_routed_batches_equal_the_routed_forward(T, block):
    """Ids through a remap table, ids as slots, and the whole forward: the same rows, bit for bit; a missing expert is
    reported and its slots own no row."""
    import blackwell_moe_b200 as bw
    D, E, K, H = 256, 16, 4, 128
    inp = make_block_inputs(T, D, E, K, H, seed=T) if block else make_inputs(T, D, E, K, H, seed=T)
    c = to_cuda(inp)
    s = "inv_" if block else "s_"
    w = (c["q_gate"], c["q_up"], c["q_down"], c[s + "gate"], c[s + "up"], c[s + "down"])
    full = bw.fp8_moe_forward(c["x"], c["w_gate"], *w, top_k=K)
    wt, idx = bw.top_k_router(c["x"], c["w_gate"], K)
    assert torch.equal(bw.fp8_moe_forward_routed(c["x"], wt, idx, *w), full)
    ids = torch.randperm(40, generator=torch.Generator().manual_seed(1))[:E].cuda()
    remap = torch.full((40,), -1, dtype=torch.int32, device="cuda")
    remap[ids] = torch.arange(E, dtype=torch.int32, device="cuda")
    named = ids[idx.long()].to(torch.int32)
    assert torch.equal(bw.fp8_moe_forward_routed(c["x"], wt, named, *w, remap=remap), full)
    gone = named.clone()
    gone[0, 1] = next(i for i in range(40) if int(remap[i]) < 0)
    bw.fp8_moe_forward_routed(c["x"], wt, gone, *w, remap=remap)
    v = bw.moe_stage_views("cuda:0", T, D, H, E, K, block=block)
    assert int(v["status"][0]) & 2 and int(v["offsets"][-1]) == T * K - 1 and int(v["pos"].view(T, K)[0, 1]) == -1


@pytest.mark.parametrize("M,E", [(1025, 7), (2048, 256), (2049, 64), (70001, 200), (524289, 16), (600000, 256)])
def test_two_pass_plan_is_the_stable_sort(M, E):
    from blackwell_moe_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M)
    ids = torch.randint(0, E, (M,), generator=g, dtype=torch.int32)
    ids[torch.randint(0, M, (5,), generator=g)] = E                     # slots that own no row
    amax = torch.rand(M, generator=g)
    i32 = lambda n, fill=-7: torch.full((n,), fill, dtype=torch.int32, device="cuda")
    offsets, pos, row_slot, row_expert, status = i32(E + 1), i32(M), i32(M), i32(M), i32(1, 0)
    seg = torch.full((E,), 9.0, device="cuda")
    scratch = torch.empty(lib.bwmoe_plan_scratch_bytes(M, E, 1), dtype=torch.uint8, device="cuda")
    d_ids, d_amax = ids.cuda(), amax.cuda()
    _lib.check(lib.bwmoe_permute_plan(d_ids.data_ptr(), d_amax.data_ptr(), M, E, 1, offsets.data_ptr(), pos.data_ptr(),
                                      row_slot.data_ptr(), row_expert.data_ptr(), seg.data_ptr(), status.data_ptr(),
                                      scratch.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    order = torch.sort(ids, stable=True).indices
    n = int((ids < E).sum())
    assert int(status[0]) == 2
    assert torch.equal(offsets.cpu().long(), torch.searchsorted(ids[order], torch.arange(E + 1, dtype=torch.int32)))
    assert torch.equal(row_slot.cpu().long()[:n], order[:n]) and torch.all(row_slot[n:] == -1)
    assert torch.equal(row_expert.cpu()[:n], ids[order[:n]]) and torch.all(row_expert[n:] == -1)
    want = torch.full((M,), -1, dtype=torch.int64)
    want[order[:n]] = torch.arange(n)
    assert torch.equal(pos.cpu().long(), want)
    ref = torch.zeros(E).scatter_reduce(0, ids[order[:n]].long(), amax[order[:n]], "amax")
    assert torch.equal(seg.cpu(), ref)


@pytest.mark.parametrize("T,D,E,K", [(8, 2048, 64, 6), (64, 1024, 256, 8), (300, 2048, 128, 8), (2000, 1024, 256, 8), (1024, 512, 8, 2)])
def test_router_with_columns_of_very_different_length(T, D, E, K):
    """Skewed popularity through a constant feature (one column several times as long as the others), tokens of zeros
    (all logits tie) and a duplicated column: still the exact order, ties to the lower id."""
    import blackwell_moe_b200 as bw
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, D, generator=g).to(BF16)
    w = (torch.randn(D, E, generator=g) * 0.02).to(BF16)
    x[:, 0] = 1.0
    w[0] = (-1.1 * torch.log(torch.randperm(E, generator=g).float() + 1.0) + 3.0).to(BF16)
    w[:, E // 2] = w[:, 1]
    x[T // 2] = 0
    wt, idx = bw.top_k_router(x.cuda(), w.cuda(), K)
    wr, ir = oracle.router_canonical(x, w, K)
    assert torch.equal(idx.cpu(), ir)
    torch.testing.assert_close(wt.cpu(), wr, rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("T,D,E,K", [(2000, 1024, 128, 8), (300, 2048, 256, 8), (1100, 512, 64, 3), (1030, 256, 16, 4)])
def test_tokens_that_one_long_column_puts_in_doubt_get_exact_weights(T, D, E, K):
    """One column is so long that, trusted to its norm, more experts than the candidate list holds might reach the K best.
    Such tokens carry the weights of the fp64 kernels bit for bit, whether their own experts' norms settle them or not."""
    import blackwell_moe_b200 as bw
    g = torch.Generator().manual_seed(D)
    x = torch.randn(T, D, generator=g).to(BF16)
    w = (torch.randn(D, E, generator=g) * 0.02).to(BF16)
    x[:, 0], w[0, E // 3] = 0.0, 250.0                   # (the feature is off: the expert's logit stays ordinary)
    wt, idx = bw.top_k_router(x.cuda(), w.cuda(), K)
    we, ie = bw.top_k_router(x.cuda(), w.cuda(), K, as_batch=32)             # the decode kernel: fp64 sums
    assert torch.equal(idx, ie)
    logits = x.double() @ w.double()
    trust = 2.0 ** -13 * x.double().norm(dim=1, keepdim=True) * w.double().norm(dim=0).max()
    near = (logits >= logits.topk(K, dim=1).values[:, -1:] - 0.95 * trust).sum(1)
    doubt = near > 12
    assert int(doubt.sum()) > T // 4
    assert torch.equal(wt.cpu()[doubt], we.cpu()[doubt])


@pytest.mark.parametrize("M,E,D,H", [(4, 4, 4096, 3584), (2, 2, 4096, 7168), (8, 8, 2048, 1408), (1, 1, 1024, 2048), (3, 5, 272, 640)])
def test_split_k_pieces_are_no_longer_than_four_rounds_of_tiles_make_them(M, E, D, H):
    """A piece is one fp32 sum of the tensor core, which truncates at every step: the longer, the less exact.  The slabs of
    the partial sums - one per piece, in scratch that starts at zero - are counted, and their sum is compared with fp64."""
    from blackwell_moe_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + H)
    hq = torch.randn(M, H, generator=g, device="cuda").to(torch.float8_e4m3fn)
    w = torch.randn(E, H, D, generator=g, device="cuda").to(torch.float8_e4m3fn)
    offsets = torch.tensor([min(e, M) for e in range(E)] + [M], dtype=torch.int32, device="cuda")
    one, status = torch.ones(E, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    y = torch.empty(M, D, dtype=BF16, device="cuda")
    scratch = torch.zeros(lib.bwmoe_gemm_scratch_bytes(M, D, H, E), dtype=torch.uint8, device="cuda")
    _lib.check(lib.bwmoe_down(hq.data_ptr(), offsets.data_ptr(), one.data_ptr(), w.data_ptr(), one.data_ptr(), M, D, H, E,
                              y.data_ptr(), status.data_ptr(), scratch.data_ptr(), torch.cuda.current_stream().cuda_stream))
    slabs = scratch[:8 * M * D * 4].view(torch.float32).view(8, M, D)
    pieces = int((slabs != 0).flatten(1).any(1).sum())
    k_blocks, tiles = -(-H // 128), min(M, E) * -(-D // 256)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    least = min(8, k_blocks // 2, -(-4 * sms // tiles))
    assert pieces >= -(-k_blocks // -(-k_blocks // least))
    assert int(status[0]) == 0
    expert = [max(e for e in range(E) if offsets[e] <= m < offsets[e + 1]) for m in range(M)]
    want = torch.stack([hq[m].double() @ w[e].double() for m, e in enumerate(expert)])
    # 4 steps per K block, each off by at most 2^-23 of a partial sum of deviation sqrt(H) or less, hardly above five times that
    assert float((slabs.double().sum(0) - want).abs().max()) < 4 * k_blocks * 2.0 ** -23 * 5 * H ** 0.5
    total = torch.zeros(M, D, device="cuda")
    for slab in slabs:
        total += slab
    assert torch.equal(y, total.to(BF16))


@pytest.mark.parametrize("T,D,K", [(1, 8, 1), (5, 264, 2), (3, 256, 5), (7, 1032, 8), (4, 512, 32), (3, 72, 33), (2, 128, 70)])
def test_combine_stage_with_ragged_rows_and_any_number_of_slots(T, D, K):
    """The combine entry point: row widths that leave lanes idle (both forms of the kernel), up to 2, 4 and 8 rows in flight,
    more slots than a warp has lanes, slots without a row - the fixed-order fp32 sum of bf16 products, bit for bit."""
    from blackwell_moe_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(T * K)
    M = T * K
    y = torch.randn(M, D, generator=g).to(BF16)
    w = torch.rand(T, K, generator=g)
    pos = torch.randperm(M, generator=g).to(torch.int32).view(T, K)
    if K > 2:
        pos[T - 1, 1] = -1
    want = torch.zeros(T, D)
    for k in range(K):
        prod = (y[pos[:, k].clamp(min=0).long()].float() * w[:, k:k + 1].to(BF16).float()).to(BF16).float()
        want += torch.where(pos[:, k:k + 1] >= 0, prod, torch.zeros(()))
    out = torch.empty(T, D, dtype=BF16, device="cuda")
    d = [t.cuda() for t in (y, pos, w)]
    _lib.check(lib.bwmoe_combine(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), T, D, K, out.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out.cpu(), want.to(BF16))


@pytest.mark.parametrize("T,E,block", [(1, 16, False), (40, 16, False), (1, 16, True), (100, 64, True), (600, 64, False)])
def test_calls_can_be_captured_and_replayed(T, E, block):
    """The launch chain (cluster launches, programmatic edges, a memset only where the tensor-core router runs) in a CUDA
    graph, behind the kernel that makes the activations: a replay on new values equals the plain call on them."""
    import blackwell_moe_b200 as bw
    D, K, H = 512, 4, 256
    inp = make_block_inputs(T, D, E, K, H, seed=T) if block else make_inputs(T, D, E, K, H, seed=T)
    c = to_cuda(inp)
    s = "inv_" if block else "s_"
    w = (c["w_gate"], c["q_gate"], c["q_up"], c["q_down"], c[s + "gate"], c[s + "up"], c[s + "down"])
    source = c["x"].clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        bw.fp8_moe_forward(source * 2, *w, top_k=K)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = bw.fp8_moe_forward(source * 2, *w, top_k=K)
    graph.replay()
    torch.cuda.synchronize()
    first = out.clone()
    for seed in (1001, 1002):
        source.copy_(torch.randn(T, D, generator=torch.Generator().manual_seed(seed)).to(BF16))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, bw.fp8_moe_forward(source * 2, *w, top_k=K))
        assert not torch.equal(out, first)
