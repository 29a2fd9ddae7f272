"""GPU tests of the individual sm_100a kernels against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    torch.cuda.set_device(0)
    return torch.device("cuda", 0)


@pytest.fixture(scope="module")
def heap(dev):
    from iris_testing_b200.parallel.symm import SymmetricHeap
    return SymmetricHeap(512 << 20)


def test_native_library_is_loaded():
    from iris_testing_b200 import _native
    lib = _native.lib()
    assert lib.b200_gemm_smem_bytes() <= 232448
    maps = open("/proc/self/maps").read()
    assert "libb200moe.so" in maps


@pytest.mark.parametrize("simple", [False, True])
@pytest.mark.parametrize("T,D,E,k,bias", [(64, 128, 8, 2, False), (1000, 256, 64, 8, False),
                                          (333, 512, 128, 4, True), (5, 64, 3, 1, False),
                                          (4096, 2048, 256, 8, True)])
def test_router_topk(dev, T, D, E, k, bias, simple):
    from iris_testing_b200.ops import cpu_ref, router_topk
    from iris_testing_b200.utils import gen_local_tokens, gen_router, zipf_expert_bias
    x = gen_local_tokens(1, T, D, torch.bfloat16, dev, 0, 0, "normal")
    wr = gen_router(D, E, torch.bfloat16, dev, 0, std=None)
    b = zipf_expert_bias(E, device=dev) if bias else None
    ref_lg = x.float() @ wr.float() + (b if bias else 0)
    if simple:
        idx, w, lg = router_topk(x, wr, k, bias=b, return_logits=True)
        assert torch.allclose(lg, ref_lg, atol=1e-4, rtol=1e-4)
    else:                                   # tensor-core path (softmax + top-k in the epilogue)
        status = torch.zeros(4, dtype=torch.int32, device=dev)
        idx, w = router_topk(x, wr, k, bias=b, status=status)
        assert status[0].item() == 0
    ridx, rw = cpu_ref.router_topk_ref(x, wr, k, bias=b)
    # near-ties may legitimately swap: compare where the reference's k-th gap is clear
    probs = torch.softmax(ref_lg, -1)
    srt = torch.sort(probs, -1, descending=True).values
    clear = (srt[:, :k] - srt[:, 1:k + 1]).min(dim=1).values > 1e-6 if E > k else torch.ones(T, dtype=torch.bool, device=dev)
    assert clear.float().mean() > 0.95
    assert torch.equal(idx[clear], ridx[clear])
    assert torch.allclose(w[clear], rw[clear], atol=1e-6, rtol=2e-4)
    _, wn = router_topk(x, wr, k, bias=b, renormalize=True, force_simple=simple)
    assert torch.allclose(wn.sum(-1), torch.ones(T, device=dev), atol=1e-5)


@pytest.mark.parametrize("T,k,E", [(64, 2, 8), (4096, 8, 128), (1, 1, 4), (1000, 4, 64)])
def test_plan_and_pack(dev, T, k, E):
    from iris_testing_b200.ops import cpu_ref, make_plan, pack_rows
    g = torch.Generator(device="cpu").manual_seed(T + k)
    idx = torch.randint(0, E, (T, k), generator=g, dtype=torch.int32).to(dev)
    if T > 100:
        idx[idx == 3] = 0                      # an empty expert and a hot one
    p = make_plan(idx, E)
    r = cpu_ref.plan_ref(idx, E)
    for name in ("counts", "bucket_start", "send_order", "dst_slot", "rank_in_bucket"):
        assert torch.equal(getattr(p, name), getattr(r, name)), name
    x = torch.randn(T, 64, device=dev).to(torch.bfloat16)
    assert torch.equal(pack_rows(x, p.send_order, k), cpu_ref.pack_ref(x, r.send_order, k))


def _gemm_case(dev, rows_list, N, K, gated, pair=False, wide=0):
    from iris_testing_b200 import _native as nv
    from iris_testing_b200.ops import grouped_gemm
    G, M = len(rows_list), max(sum(rows_list), 1)
    g = torch.Generator(device="cpu").manual_seed(N + K)
    a = torch.randn(M, K, generator=g).to(dev, torch.bfloat16)
    w = (torch.randn(G, N, K, generator=g) * 0.05).to(dev, torch.bfloat16)
    rows = torch.tensor(rows_list, dtype=torch.int32, device=dev)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    out = grouped_gemm(a, w, rows, epilogue=nv.EPI_SILU_GATE if gated else nv.EPI_STORE, status=status,
                       cta_pair=pair, wide_tiles=wide)
    ref = torch.zeros(M, N, device=dev)
    off = 0
    for gi, r in enumerate(rows_list):
        ref[off:off + r] = a[off:off + r].float() @ w[gi].float().t()
        off += r
    if gated:
        v = ref.view(M, N // 256, 2, 128)
        ref = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(M, N // 2)
    n = sum(rows_list)
    assert status[0].item() == 0
    assert torch.allclose(out[:n].float(), ref[:n], atol=2e-2 * float(ref.abs().max()) + 1e-3, rtol=2e-2)


@pytest.mark.parametrize("rows,N,K", [([128], 256, 64), ([100], 256, 512), ([300, 0, 77, 129], 512, 512),
                                      ([37] * 16, 2048, 1408), ([5, 200], 136, 72), ([0, 0, 1], 256, 128),
                                      ([4096], 1024, 4096)])
@pytest.mark.parametrize("pair", [False, True])
def test_grouped_gemm_plain(dev, rows, N, K, pair):
    _gemm_case(dev, rows, N, K, gated=False, pair=pair)


@pytest.mark.parametrize("rows,N,K", [([300, 0, 77, 129], 512, 512), ([1000, 513], 2816, 2048)])
@pytest.mark.parametrize("pair", [False, True])
def test_grouped_gemm_silu_gate(dev, rows, N, K, pair):
    _gemm_case(dev, rows, N, K, gated=True, pair=pair)


@pytest.mark.parametrize("rows,N,K,gated", [([300, 0, 77, 129], 512, 512, False), ([4096], 1024, 4096, False),
                                            ([1000, 513], 2816, 2048, True), ([700], 768, 256, False),
                                            ([37] * 16, 2048, 1408, False), ([256, 255, 257], 1280, 64, True),
                                            ([5000], 136, 72, False)])
def test_grouped_gemm_wide_tiles(dev, rows, N, K, gated):
    """512-column tiles (both TMEM accumulators per tile, second half's MMAs trailing the first):
    also with an odd number of 256-column blocks, where the last tile's second half is past N."""
    _gemm_case(dev, rows, N, K, gated=gated, pair=True, wide=1)


def test_expert_op_reference_signature(dev):
    """Oracle of the reference's dead test_gemm (unit_tests.py:224-237): per-expert matmul, tol 1e-2."""
    from iris_testing_b200.ops import expert
    from iris_testing_b200.utils import gen_local_weights
    g = torch.Generator(device="cpu").manual_seed(0)
    cnt = torch.randint(0, 100, (6,), generator=g, dtype=torch.int32)
    S = int(cnt.sum())
    tokens = torch.randn(S, 128, generator=g).to(dev, torch.bfloat16)
    w = gen_local_weights(6, 128, 256, torch.bfloat16, dev, 0, 0)
    out = expert(tokens, w, cnt.to(dev))
    off = 0
    for e, n in enumerate(cnt.tolist()):
        ref = tokens[off:off + n].float() @ w[e].float()
        assert torch.allclose(out[off:off + n].float(), ref, atol=1e-2, rtol=1e-2)
        off += n


def test_silu_gate(dev):
    from iris_testing_b200.ops import silu_gate
    g, u = torch.randn(513, 256, device=dev).bfloat16(), torch.randn(513, 256, device=dev).bfloat16()
    ref = torch.nn.functional.silu(g.float()) * u.float()
    assert torch.allclose(silu_gate(g, u).float(), ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("e_local,H,cap", [(2, 128, 32), (4, 256, 16)])
def test_custom_a2a_reference_unit_shapes(dev, heap, e_local, H, cap):
    """The reference's two unit-test shapes (unit_tests.py:84-88) on a world of one: full
    routing, value-encodes-coordinates payload, exact equality per (src, e) block."""
    from iris_testing_b200.ops import custom_a2a, shuffle, unshuffle
    from iris_testing_b200.utils import (alloc_shmem_buffers, build_dst_offsets, expected_tiles,
                                         reset_dispatch_flags, spin_wait_counts_ready,
                                         spin_wait_token_sync)
    world = 1
    counts = torch.full((world, e_local), cap, dtype=torch.int32, device=dev)
    t = torch.arange(cap, device=dev).view(1, cap, 1)
    e = torch.arange(e_local, device=dev).view(e_local, 1, 1)
    payload = (e * 100 + t).expand(e_local, cap, H).reshape(-1, H).to(torch.bfloat16).contiguous()
    b = alloc_shmem_buffers(heap, world, e_local, cap, H, torch.bfloat16)
    for _ in range(2):                      # second call after the reference's flag reset
        reset_dispatch_flags(b)
        out = custom_a2a(payload, counts, build_dst_offsets(counts), b.pca, b.token_buf,
                         b.counts_ready, b.token_sync, b.heap_bases, e_local * world, cap)
        spin_wait_counts_ready(b.counts_ready, world, timeout_s=5)
        spin_wait_token_sync(b.token_sync, expected_tiles(b.pca, 32), timeout_s=5)
        assert torch.equal(b.pca, counts.t())
        assert torch.equal(out.view(-1, H), payload)
    packed, rows = shuffle(b.token_buf, b.pca, b.token_sync, b.counts_ready)
    assert rows.tolist() == [cap] * e_local and torch.equal(packed, payload)
    assert torch.equal(unshuffle(packed, b.pca, cap), b.token_buf)
    heap.check_status()


def test_unfused_pipeline_ragged_single_gpu(dev, heap):
    """Router-driven ragged counts through dispatch -> shuffle -> expert -> unshuffle -> return ->
    weighted sum, against the dense reference; padding rows stay zero; overflow is reported."""
    from iris_testing_b200.ops import cpu_ref, custom_a2a, expert, shuffle, unshuffle
    from iris_testing_b200.ops.combine import padded_return, weighted_gather
    from iris_testing_b200.utils import (alloc_return_buffers, alloc_shmem_buffers, gen_local_tokens,
                                         gen_local_weights, gen_router, route_and_pack)
    D, E, k, T = 256, 8, 2, 300
    x = gen_local_tokens(1, T, D, torch.bfloat16, dev, 1, 0, "normal")
    router = gen_router(D, E, torch.bfloat16, dev, 1, std=None)
    w = gen_local_weights(E, D, D, torch.bfloat16, dev, 1, 0, std=0.05)
    payload, counts, dst_off, _, idx, wgt, plan = route_and_pack(x, router, k, 1, E)
    cap = int(counts.max().item())
    guard_lo = heap.zeros((4096,), torch.int32); guard_lo.fill_(0x5A5A5A5A)     # canaries around the
    b = alloc_shmem_buffers(heap, 1, E, cap, D, torch.bfloat16)                   # symmetric buffers
    guard_hi = heap.zeros((4096,), torch.int32); guard_hi.fill_(0x5A5A5A5A)
    custom_a2a(payload, counts, dst_off, b.pca, b.token_buf, b.counts_ready, b.token_sync,
               b.heap_bases, E, cap)
    packed, rows = shuffle(b.token_buf, b.pca, b.token_sync, b.counts_ready)
    n = int(rows.sum().item())
    assert torch.equal(packed[:n], payload)                 # world of one: same order
    valid = torch.arange(cap, device=dev).view(1, 1, cap) < b.pca.unsqueeze(-1)
    assert float(b.token_buf[~valid].abs().sum()) == 0.0     # padding is zero
    out = expert(packed, w, rows)
    out_buf = unshuffle(out, b.pca, cap)
    r = alloc_return_buffers(heap, 1, E, cap, D, torch.bfloat16)
    padded_return(out_buf, b.pca, r.ret_buf, r.ret_sync, b.heap_bases)
    y = weighted_gather(r.ret_buf, plan, idx, wgt, r.ret_sync, 1, cap, status=heap.status)
    ref = cpu_ref.dense_moe_ref(x, router, k, w_single=w)
    assert torch.allclose(y.float(), ref, atol=2e-2 * float(ref.abs().max()), rtol=2e-2)
    heap.check_status()
    assert bool((guard_lo == 0x5A5A5A5A).all()) and bool((guard_hi == 0x5A5A5A5A).all())
    # capacity too small: rows beyond CAP are dropped and the status word says so
    small = alloc_shmem_buffers(heap, 1, E, max(cap // 2, 1), D, torch.bfloat16)
    custom_a2a(payload, counts, dst_off, small.pca, small.token_buf, small.counts_ready,
               small.token_sync, small.heap_bases, E, max(cap // 2, 1))
    torch.cuda.synchronize()
    with pytest.raises(Exception, match="overflow"):
        heap.check_status()


def test_heap_barrier_and_bounded_wait(dev, heap):
    heap.barrier()
    heap.barrier()
    # a wait that nothing satisfies must return with a status, not hang
    from iris_testing_b200.ops import shuffle
    pca = torch.full((2, 1), 4, dtype=torch.int32, device=dev)
    buf = torch.zeros(2, 1, 4, 64, dtype=torch.bfloat16, device=dev)
    never = torch.zeros(2, dtype=torch.int32, device=dev)
    ready = torch.ones(1, dtype=torch.int32, device=dev)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    shuffle(buf, pca, never, ready, status=status, wait_budget_ms=50)
    torch.cuda.synchronize()
    assert status[0].item() == 6     # "a dispatched token tile never arrived"


def test_device_row_counts_beyond_the_buffers_are_reported_not_stored(dev):
    """Row counts are read on the device; counts that add up to more rows than a buffer holds
    must end in a status code, never in a store past the buffer."""
    from iris_testing_b200.ops import check_default_status, default_status, grouped_gemm, shuffle
    a = torch.randn(256, 128, device=dev).to(torch.bfloat16)
    w = torch.randn(2, 256, 128, device=dev).to(torch.bfloat16)
    out = torch.zeros(256 + 64, 256, dtype=torch.bfloat16, device=dev)       # 64 guard rows behind the output
    rows = torch.tensor([200, 200], dtype=torch.int32, device=dev)           # 400 > 256
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    grouped_gemm(a, w, rows, out=out[:256], status=status)
    torch.cuda.synchronize()
    assert status.tolist()[:2] == [10, 400] and float(out.abs().sum()) == 0.0
    # same call without a status tensor: the report lands in the device's default status word
    default_status(dev).zero_()
    grouped_gemm(a, w, rows, out=out[:256])
    with pytest.raises(Exception, match=r"overflow.*rows needed: 400"):
        check_default_status(dev)
    check_default_status(dev)                                                # reset by the failed check
    # shuffle into a packed buffer that is too small: the copy stops at max_rows
    pca = torch.tensor([[6], [5]], dtype=torch.int32, device=dev)
    buf = torch.ones(2, 1, 8, 64, dtype=torch.bfloat16, device=dev)
    st2 = torch.zeros(4, dtype=torch.int32, device=dev)
    packed, _ = shuffle(buf, pca, max_rows=8, status=st2)
    torch.cuda.synchronize()
    assert packed.shape[0] == 8 and st2.tolist()[:2] == [10, 11]


@pytest.mark.parametrize("mode", ["stores", "bulk"])
@pytest.mark.parametrize("e_local,H,T,k,combine", [(2, 128, 100, 2, False), (8, 4096, 1024, 2, True),
                                                   (4, 768, 777, 4, True), (1, 264, 50, 1, True)])
def test_padded_all_to_all_engine_repeats_without_memsets(dev, e_local, H, T, k, combine, mode):
    """``PaddedAllToAll`` on a world of one, three exchanges in a row with changing routing: flags
    re-armed in-kernel, valid rows bit-equal to the payload, padding never written, and with
    the return path the weighted sum of the rows that come home."""
    from iris_testing_b200.parallel.padded_a2a import CapacityProbe, PaddedAllToAll
    from iris_testing_b200.parallel.symm import SymmetricHeap
    from iris_testing_b200.utils import gen_local_tokens, gen_router, route_and_pack
    E = e_local
    heap = SymmetricHeap(64 << 20, max_bytes=1 << 30)
    probe = CapacityProbe(heap, e_local)
    router = gen_router(H, E, torch.bfloat16, dev, 3, std=None)
    xs = [gen_local_tokens(1, T, H, torch.bfloat16, dev, s, 0, "normal") for s in range(3)]
    routed = [route_and_pack(x, router, k, 1, E) for x in xs]
    caps = torch.stack([probe.measure(r[1].contiguous()) for r in routed]).tolist()
    for c, r in zip(caps, routed):
        n = r[1].to(torch.int64)
        assert c == [int(n.max()), int(n.sum()), int(n.sum()), int(n.sum())]     # CAP, M, rows received
    cap = max(c[0] for c in caps)
    a2a = PaddedAllToAll(heap, e_local, cap, H, torch.bfloat16, with_return=combine, copy_mode=mode)
    a2a.token_buf.fill_(7.0)                                  # rows no exchange has used stay as they were
    high = torch.zeros(e_local, dtype=torch.int64)            # most rows each cell has ever held
    for x, (payload, counts, dst_off, _, idx, wgt, plan) in zip(xs, routed):
        out = a2a.dispatch(payload, counts, dst_off)
        a2a.wait()
        torch.cuda.synchronize()
        assert torch.equal(a2a.pca, counts.t()) and int(a2a.counts_ready[0]) == 1
        tiles = ((counts.reshape(-1) + 31) // 32).to(torch.int32)
        assert torch.equal(a2a.token_sync, tiles)
        off = 0
        for e, n in enumerate(counts.reshape(-1).tolist()):
            assert torch.equal(out[e, 0, :n], payload[off:off + n]), e
            high[e] = max(int(high[e]), n)
            assert float((out[e, 0, int(high[e]):].float() - 7.0).abs().sum()) == 0.0   # never written
            off += n
        if combine:
            a2a.send_back()
            y = a2a.reduce(plan, idx, wgt)
            ref = x.float() * wgt.sum(dim=1, keepdim=True)
            assert torch.allclose(y.float(), ref, atol=2e-2 * float(ref.abs().max()), rtol=2e-2)
            torch.cuda.synchronize()
            assert int(a2a.ret.ret_sync.abs().sum()) == 0     # re-armed by the reduce
    heap.check_status()
    del a2a, probe
    heap.close()


@pytest.mark.parametrize("T,D,E,k", [(1, 8, 1, 1), (15, 72, 8, 2), (16, 64, 9, 8), (17, 136, 16, 4), (33, 1000, 17, 2),
                                     (31, 2048, 33, 8), (9471, 72, 8, 2), (9472, 72, 16, 2), (9473, 136, 32, 4),
                                     (9500, 200, 65, 8), (40, 4096, 256, 8),
                                     (4736, 64, 64, 8), (4737, 64, 64, 8)])
def test_router_tile_edges(dev, T, D, E, k):
    """Batches around one 128-token tile's edges and of many tiles, last k-blocks of any length, and one to
    sixteen 16-column steps of experts."""
    from iris_testing_b200.ops import cpu_ref, router_topk
    from iris_testing_b200.utils import gen_local_tokens, gen_router
    x = gen_local_tokens(1, T, D, torch.bfloat16, dev, 1, 0, "normal")
    wr = gen_router(D, E, torch.bfloat16, dev, 1, std=None)
    idx, w = router_topk(x, wr, k)
    ridx, rw = cpu_ref.router_topk_ref(x, wr, k)
    clear = cpu_ref.clear_routing_mask(x, wr, k, None)
    assert clear.float().mean() > 0.95
    assert torch.equal(idx[clear], ridx[clear])
    assert torch.allclose(w[clear], rw[clear], atol=1e-6, rtol=2e-4)      # fp32 sums of up to 4096 products


@pytest.mark.parametrize("D,E,k,T", [(4096, 8, 2, 2400), (2048, 64, 8, 4800), (1024, 32, 2, 9600)])
def test_a_token_is_routed_alike_in_every_batch(dev, D, E, k, T):
    """Choices and weights of a token are the same bits whatever batch it comes in: near-ties of two logits
    are decided by the summation order, which must not change with the number of tokens."""
    from iris_testing_b200.ops import router_topk
    from iris_testing_b200.utils import gen_local_tokens, gen_router
    x = gen_local_tokens(1, T, D, torch.bfloat16, dev, 5, 0, "normal")
    wr = gen_router(D, E, torch.bfloat16, dev, 5, std=None)
    idx, w = router_topk(x, wr, k)
    for n in (1, 17, 200, T // 2 - 64, T - 1):
        i, v = router_topk(x[:n], wr, k)
        assert torch.equal(i, idx[:n]) and torch.equal(v, w[:n]), n


def test_small_route_and_plan_from_several_threads(dev):
    """Host threads with other numbers of experts in the same kernel: no launch is refused and every result is that
    of the call alone."""
    import ctypes as C
    import threading
    from iris_testing_b200.ops import cpu_ref
    from iris_testing_b200.ops._common import declare
    from iris_testing_b200.ops.plan import PlanPushArgs
    from iris_testing_b200.ops.router import router_kmajor
    from iris_testing_b200.utils import gen_local_tokens, gen_router
    fn = declare("b200_route_plan_small",
                 [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p,
                  C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.POINTER(PlanPushArgs), C.c_void_p, C.c_void_p])
    T, D, k, errors = 48, 64, 2, []

    def work(E):
        i32 = dict(dtype=torch.int32, device=dev)
        x = gen_local_tokens(1, T, D, torch.bfloat16, dev, E, 0, "normal")
        wr = gen_router(D, E, torch.bfloat16, dev, E, std=None)
        wk = router_kmajor(wr)
        idx, w = torch.empty(T, k, **i32), torch.empty(T, k, dtype=torch.float32, device=dev)
        outs = [torch.empty(n, **i32) for n in (E, E + 1, T * k, T * k)]
        ticket = torch.zeros(1, **i32)
        stream = torch.cuda.Stream(dev)
        torch.cuda.synchronize()
        for _ in range(2000):
            rc = fn(x.data_ptr(), wk.data_ptr(), None, T, D, E, k, 0, idx.data_ptr(), w.data_ptr(),
                    *(t.data_ptr() for t in outs), None, ticket.data_ptr(), stream.cuda_stream)
            if rc != 0:
                errors.append((E, rc))
                break
        stream.synchronize()
        ref = cpu_ref.router_topk_ref(x, wr, k)[0]
        plan = cpu_ref.plan_ref(idx, E)
        clear = cpu_ref.clear_routing_mask(x, wr, k, None)
        if not errors and not (torch.equal(idx[clear], ref[clear]) and torch.equal(outs[0], plan.counts)
                               and torch.equal(outs[2], plan.send_order) and torch.equal(outs[3], plan.dst_slot)):
            errors.append((E, "wrong"))

    work(40), work(128)                                  # settled before the threads start
    threads = [threading.Thread(target=work, args=(E,)) for E in (40, 128, 64)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("n,E", [(0, 4), (1, 128), (1023, 3), (1024, 128), (1025, 1), (148 * 1024, 64),
                                 (148 * 1024 + 1, 128), (400000, 8)])
def test_plan_chunk_edges(dev, n, E):
    """Lists around one chunk of the plan kernels, around all chunks of one pass, and of several passes."""
    from iris_testing_b200.ops import cpu_ref, make_plan
    g = torch.Generator(device="cpu").manual_seed(n + E)
    idx = torch.randint(0, E, (n, 1), generator=g, dtype=torch.int32).to(dev)
    p, r = make_plan(idx, E), cpu_ref.plan_ref(idx, E)
    for name in ("counts", "bucket_start", "send_order", "dst_slot", "rank_in_bucket"):
        assert torch.equal(getattr(p, name), getattr(r, name)), name


def test_plan_refuses_a_short_workspace(dev):
    from iris_testing_b200.ops import make_plan
    from iris_testing_b200.ops.plan import plan_workspace
    idx = torch.zeros((4, 2), dtype=torch.int32, device=dev)
    with pytest.raises(ValueError, match="workspace"):
        make_plan(idx, 16, workspace=plan_workspace(8, dev))
    assert make_plan(idx, 8, workspace=plan_workspace(16, dev)).counts.tolist() == [8] + [0] * 7


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (5, 2, 4), (600, 3, 8), (40000, 4, 128)])
def test_plan_and_its_users_drop_copies_without_an_expert(dev, T, k, E):
    """Expert numbers below zero and past the last: no place for the copy, -1 behind the send order's last row, a zero
    payload row, no part in the weighted sum; with none left at all too.  Both plan entry points."""
    from iris_testing_b200 import _native as nv
    from iris_testing_b200.ops import cpu_ref, make_plan
    from iris_testing_b200.ops._common import ptr, stream_ptr
    from iris_testing_b200.ops.combine import weighted_gather
    from iris_testing_b200.ops.plan import pack_rows
    g = torch.Generator(device="cpu").manual_seed(T + E)
    H = 72
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(dev)
    for lo, hi in ((-1, E), (-3, E + 3), (-1, 0)):
        idx = torch.randint(lo, hi, (T, k), generator=g, dtype=torch.int32).to(dev)
        p, r = make_plan(idx, E), cpu_ref.plan_ref(idx, E)
        for name in ("counts", "bucket_start", "send_order", "dst_slot", "rank_in_bucket"):
            assert torch.equal(getattr(p, name), getattr(r, name)), name
        q = {n: torch.full_like(getattr(r, n), 12345) for n in ("counts", "bucket_start", "send_order", "dst_slot")}
        assert nv.lib().b200_plan_noalloc(ptr(idx), T * k, E, *(ptr(t) for t in q.values()), stream_ptr(idx)) == 0
        for name, t in q.items():
            assert torch.equal(t, getattr(r, name)), name
        payload = pack_rows(x, p.send_order, k)
        assert torch.equal(payload, cpu_ref.pack_ref(x, r.send_order, k))
        cap = max(int(p.counts.max()), 1)
        ret = torch.zeros(1, E, cap, H, dtype=torch.bfloat16, device=dev)
        for e, (a, n) in enumerate(zip(p.bucket_start.tolist(), p.counts.tolist())):
            ret[0, e, :n] = payload[a:a + n]
        keep = (idx >= 0) & (idx < E)
        w = torch.where(keep, torch.rand(T, k, generator=g).to(dev), float("nan"))
        y = weighted_gather(ret, p, idx, w, None, 1, cap)
        sums = torch.where(keep, w, 0.0).double().sum(1, keepdim=True)
        mag = x.double().abs() * sums                    # bf16 rounding, fp32 sums of k products
        assert bool(((y.double() - x.double() * sums).abs() <= mag * (2.0 ** -8 + k * 2.0 ** -22)).all())


def test_a_token_of_nan_disturbs_no_other(dev):
    """Route, pack, dispatch, return and weighted sum with NaN tokens and masked experts: their copies are dropped and
    every other token comes back as it would alone."""
    from iris_testing_b200.ops import router_topk
    from iris_testing_b200.parallel.padded_a2a import PaddedAllToAll
    from iris_testing_b200.parallel.symm import SymmetricHeap
    from iris_testing_b200.utils import gen_local_tokens, gen_router, route_and_pack
    T, H, E, k = 300, 136, 8, 2
    x = gen_local_tokens(1, T, H, torch.bfloat16, dev, 1, 0, "normal")
    router = gen_router(H, E, torch.bfloat16, dev, 3, std=None)
    clean_idx, clean_w = router_topk(x, router, k)
    bad = torch.zeros(T, dtype=torch.bool, device=dev)
    bad[::7] = True
    x[bad] = float("nan")
    payload, counts, dst_off, _, idx, wgt, plan = route_and_pack(x, router, k, 1, E)
    assert bool((idx[bad] == -1).all()) and torch.equal(idx[~bad], clean_idx[~bad]) and torch.equal(wgt[~bad], clean_w[~bad])
    assert int(counts.sum()) == int((~bad).sum()) * k and bool(torch.isfinite(payload).all())
    heap = SymmetricHeap(2 * E * T * H * 2 + (32 << 20))
    a2a = PaddedAllToAll(heap, E, T, H, torch.bfloat16, with_return=True)
    a2a.dispatch(payload, counts, dst_off)
    a2a.wait()
    a2a.send_back()
    y = a2a.reduce(plan, idx, wgt)
    heap.check_status()
    ref = x.double() * wgt.double().sum(1, keepdim=True)
    assert int(y[bad].abs().sum()) == 0
    assert bool(((y.double() - ref).abs()[~bad] <= ref.abs()[~bad] * (2.0 ** -8 + k * 2.0 ** -22)).all())
    bias = torch.full((E,), -float("inf"), device=dev)
    bias[5] = 0.0                                        # one expert left of two asked for
    idx, wgt = router_topk(x[~bad], router, k, bias=bias)
    assert bool((idx == torch.tensor([5, -1], device=dev)).all()) and bool((wgt == torch.tensor([1.0, 0.0], device=dev)).all())
    del a2a
    heap.close()


@pytest.mark.parametrize("G,K,N", [(1, 8, 8), (2, 64, 64), (3, 72, 200), (2, 136, 56), (32, 768, 768)])
def test_weight_transpose_kernel(dev, G, K, N):
    from iris_testing_b200.ops.expert import _to_kmajor_cuda as to_kmajor
    w = torch.randn(G, K, N, device=dev).to(torch.bfloat16)
    assert torch.equal(to_kmajor(w), w.transpose(1, 2).contiguous())
    assert torch.equal(to_kmajor(w[:, :, : N // 2 + 1]), w[:, :, : N // 2 + 1].transpose(1, 2))   # general path


@pytest.mark.parametrize("T,k,E,H,drop", [(1, 1, 2, 8, False), (33, 2, 4, 264, True), (100, 3, 8, 520, False),
                                          (65, 5, 8, 2048, True), (40, 11, 16, 72, False)])
def test_weighted_gather_row_groups(dev, T, k, E, H, drop):
    """Rows in groups of 2, 4 and 8 (more slots than a group too), ragged last column pieces, dropped rows.
    Sums of k products in fp32 rounded to bf16: within one bf16 step of the fp32 result."""
    from iris_testing_b200.ops import make_plan
    from iris_testing_b200.ops.combine import weighted_gather
    g = torch.Generator(device="cpu").manual_seed(T + k)
    idx = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).to(torch.int32).to(dev)
    plan = make_plan(idx, E)
    cap = max(int(plan.counts.max()) - (3 if drop else 0), 1)
    ret = torch.randn(1, E, cap, H, device=dev).to(torch.bfloat16)
    w = torch.rand(T, k, device=dev)
    y = weighted_gather(ret, plan, idx, w, None, 1, cap)
    m = plan.dst_slot.long() - plan.bucket_start.long()[idx.reshape(-1).long()]
    rows = ret.reshape(-1, H).double()[idx.reshape(-1).long() * cap + m.clamp(max=cap - 1)]
    ref = (rows * (w.reshape(-1, 1).double() * (m < cap).unsqueeze(1))).view(T, k, H).sum(1)
    mag = (rows.abs() * w.reshape(-1, 1).double()).view(T, k, H).sum(1)
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * k * 2.0 ** -23).all())


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (33, 2, 136), (300, 2, 4096), (2400, 2, 264), (4800, 2, 72), (9500, 2, 64)])
def test_padded_exchange_shares_of_tiles(dev, T, k, H):
    """Tiles shared by eight, four and two blocks and by none, another share count from call to call, a
    dispatch whose return is left out: rows bit-equal, every tile counted once."""
    from iris_testing_b200.parallel.padded_a2a import PaddedAllToAll
    from iris_testing_b200.parallel.symm import SymmetricHeap
    from iris_testing_b200.utils import gen_local_tokens, gen_router, route_and_pack
    E = 4
    heap = SymmetricHeap(2 * E * T * H * 2 + (32 << 20))
    a2a = PaddedAllToAll(heap, E, T, H, torch.bfloat16, with_return=True)
    router = gen_router(H, E, torch.bfloat16, dev, 3, std=None)
    for i, n in enumerate((T, max(T // 9, 1), T, T)):
        x = gen_local_tokens(1, n, H, torch.bfloat16, dev, i, 0, "normal")
        payload, counts, dst_off, _, idx, wgt, plan = route_and_pack(x, router, k, 1, E)
        out = a2a.dispatch(payload, counts, dst_off)
        a2a.wait()
        assert torch.equal(a2a.token_sync, ((counts.reshape(-1) + 31) // 32).to(torch.int32))
        cells = torch.cat([out[e, 0, :c] for e, c in enumerate(counts.reshape(-1).tolist())])
        assert torch.equal(cells, payload)
        if i != 1:
            a2a.send_back()
            y = a2a.reduce(plan, idx, wgt)
            back = torch.cat([a2a.ret.ret_buf[0, e, :c] for e, c in enumerate(counts.reshape(-1).tolist())])
            assert torch.equal(back, payload) and int(a2a.ret.ret_sync.abs().sum()) == 0
            ref = x.double() * wgt.double().sum(1, keepdim=True)
            mag = x.double().abs() * wgt.double().sum(1, keepdim=True)     # bf16 rounding, fp32 sums of k products
            assert bool(((y.double() - ref).abs() <= mag * (2.0 ** -8 + k * 2.0 ** -22)).all())
        assert int(a2a._parts.abs().sum()) == 0
    heap.check_status()
    del a2a
    heap.close()
