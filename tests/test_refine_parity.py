"""The refinement kernel (``pa_refine``: stage 2 on the sub-graph, stage 3 on the
full graph, visited marks from the device pool) against

* the CPU oracle restating upstream ``traverse_refine`` with THIS kernel's
  summation order: ids, distance bits and per-stage counters identical;
* upstream's own ``traverse_refine`` (AVX2 order, built with -ffast-math, so no
  bit equality): top-k ids identical for at least 99.5 % of the queries,
  distances within 1e-5 relative.

The handoff both sides consume is produced by the traversal kernel of this
package on the same tensors.
"""
import os

import pytest
import torch

from helpers import make_problem, to_cuda

pytestmark = pytest.mark.gpu


def _case(n=12000, d=96, d_p=32, ratio=0.5, batch=256, ef=48, law="powerlaw", seed=41,
          n_init=32):
    """Handoff [B, 4*ef] from the reduced-space traversal + everything the
    refinement needs, CPU and CUDA."""
    from pilotann_b200 import extension
    p = make_problem(n=n, d=d, ratio=ratio, batch=batch, n_init=n_init, seed=seed, law=law,
                     build_device="cuda")
    full = p["full"]
    reduced = p["storage"][:, :d_p].contiguous()              # rows of the sampled nodes
    q = p["query"]
    q_red = q[:, :d_p].contiguous()
    g = torch.Generator().manual_seed(seed)
    ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (batch, n_init), generator=g)]
    diff = q_red.unsqueeze(1) - full[ids][:, :, :d_p]
    init_D = (diff * diff).sum(-1).contiguous()
    dev = "cuda"
    nbr, row_of = extension.pack_graph(p["indptr"].to(dev), p["indices"].to(dev),
                                       p["mapping"].to(dev), reduced.size(0), 32)
    oI = torch.empty(batch, 4, ef, dtype=torch.int64, device=dev)
    oD = torch.empty(batch, 4, ef, device=dev)
    extension.traverse_packed(oI, oD, nbr, row_of, reduced.to(dev), q_red.to(dev), ids.to(dev),
                              init_D.to(dev), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].to(dev), p["full_indices"].to(dev), 32)
    torch.cuda.synchronize()
    return dict(p=p, nbr=nbr, row_of=row_of, full_nbr=full_nbr, hand_I=oI, hand_D=oD,
                full=full, full_cuda=full.to(dev), q=q, q_cuda=q.to(dev), d_p=d_p, ef=ef)


@pytest.mark.parametrize("ef,d,d_p,law", [(16, 64, 32, "fuzz"), (48, 96, 32, "powerlaw"),
                                          (128, 200, 96, "powerlaw-ood"), (40, 64, 64, "mixture")])
def test_both_stages_bit_exact_vs_oracle(oracle_lib, ef, d, d_p, law):
    from pilotann_b200 import extension
    c = _case(d=d, d_p=d_p, ef=ef, law=law, batch=192)
    p = c["p"]
    k = 10
    pool = extension.VisitedPool(c["full"].size(0), 96)      # fewer slots than queries
    sub = [p["indptr"], p["indices"]]
    full = [p["full_indptr"], p["full_indices"]]
    hI = c["hand_I"].reshape(192, -1).cpu()
    hD = c["hand_D"].reshape(192, -1).cpu()
    # stage 2 alone: the rewritten handoff rows
    st = torch.zeros(192, 4, dtype=torch.int32, device="cuda")
    g_I, g_D = extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"],
                                c["row_of"], None, pool, ef, d_p, k=None, stats=st)
    w_bI, w_bD = hI.clone(), hD.clone()
    _, _, w_st = oracle_lib.refine_ex(w_bI, w_bD, sub, full, c["full"], c["q"], k, ef, d_p,
                                      gpu_order=True, stages=2, with_stats=True)
    torch.cuda.synchronize()
    assert torch.equal(g_I.cpu(), w_bI)
    assert torch.equal(g_D.cpu().view(torch.int32), w_bD.view(torch.int32))
    assert torch.equal(st.cpu()[:, :2], w_st[:, :2])
    H = oracle_lib.cpu_heap_size_for(ef)
    assert (g_I[:, : 4 * ef - H] == -1).all() and (g_I[:, -1] >= 0).float().mean() > 0.9
    # both stages: top-k
    st.zero_()
    t_I, t_D = extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"],
                                c["row_of"], c["full_nbr"], pool, ef, d_p, k=k, stats=st)
    w_I, w_D, w_st = oracle_lib.refine_ex(hI.clone(), hD.clone(), sub, full, c["full"], c["q"], k,
                                          ef, d_p, gpu_order=True, stages=3, with_stats=True)
    torch.cuda.synchronize()
    assert torch.equal(t_I.cpu(), w_I)
    assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))
    assert torch.equal(st.cpu(), w_st)
    # the handoff itself was only read
    assert torch.equal(c["hand_I"].reshape(192, -1).cpu(), hI)
    # exact distances of what came back
    exact = (c["q"].unsqueeze(1) - c["full"][w_I]).square().sum(-1)
    assert torch.allclose(t_D.cpu(), exact, rtol=1e-4, atol=1e-6)


def test_against_upstream_traverse_refine(ref_ext):
    from pilotann_b200 import extension, utils
    ef, k = 64, 10
    c = _case(n=20000, d=128, d_p=32, ef=ef, law="powerlaw", batch=512, seed=43)
    p = c["p"]
    B = 512
    pool = extension.VisitedPool(c["full"].size(0), 1024)
    t_I, t_D = extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"],
                                c["row_of"], c["full_nbr"], pool, ef, c["d_p"], k=k)
    torch.cuda.synchronize()
    hI = c["hand_I"].reshape(B, -1).cpu().clone()
    hD = c["hand_D"].reshape(B, -1).cpu().clone()
    u_I = torch.empty(B, k, dtype=torch.int64)
    u_D = torch.empty(B, k, dtype=torch.float32)
    ref_ext.traverse_refine(u_I, u_D, hI, hD, hI, hD, [p["indptr"], p["indices"]],
                            [p["full_indptr"], p["full_indices"]], c["full"], c["q"], ef, c["d_p"])
    same = (t_I.cpu() == u_I).all(dim=1).float().mean().item()
    print(f"top-{k} rows identical to upstream traverse_refine: {same:.4f}")
    assert same >= 0.995
    both = t_I.cpu() == u_I
    rel = ((t_D.cpu() - u_D).abs() / u_D.abs().clamp_min(1e-30))[both]
    assert rel.max().item() <= 1e-5
    truth = utils.ground_truth(c["q"], c["full"], k)
    assert abs(utils.recall(t_I.cpu(), truth) - utils.recall(u_I, truth)) <= 0.002
    # stage 2 alone, then upstream's full-graph search on its rows: what a caller
    # gets who keeps stage 3 on the CPU
    s_I, s_D = extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"],
                                c["row_of"], None, pool, ef, c["d_p"], k=None)
    v_I = torch.empty(B, k, dtype=torch.int64)
    v_D = torch.empty(B, k, dtype=torch.float32)
    ref_ext.traverse_cpu(v_I, v_D, s_I.cpu(), s_D.cpu(), p["full_indptr"], p["full_indices"],
                         c["full"], c["q"], ef)
    assert abs(utils.recall(v_I, truth) - utils.recall(u_I, truth)) <= 0.005
    # after upstream's stage 2 the buffer holds exact full distances
    # (test/kernel/test_traverse_refine.py:89-95 checks the same of upstream)
    real = s_I.cpu() >= 0
    exact = (c["q"].unsqueeze(1) - c["full"][s_I.cpu().clamp_min(0)]).square().sum(-1)
    assert torch.allclose(s_D.cpu()[real], exact[real], rtol=1e-4, atol=1e-6)


def test_marker_wrap_and_slot_reuse(oracle_lib):
    """One slot serves 600 queries in a row: its marker passes 254 twice and the
    array is wiped in between; results stay those of the oracle."""
    from pilotann_b200 import extension
    ef, k, B = 16, 5, 600
    c = _case(n=6000, d=64, d_p=32, ef=ef, law="fuzz", batch=B, seed=47)
    p = c["p"]
    pool = extension.VisitedPool(c["full"].size(0), 1)
    t_I, t_D = extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"],
                                c["row_of"], c["full_nbr"], pool, ef, c["d_p"], k=k)
    torch.cuda.synchronize()
    w_I, w_D = oracle_lib.refine_ex(c["hand_I"].reshape(B, -1).cpu().clone(),
                                    c["hand_D"].reshape(B, -1).cpu().clone(),
                                    [p["indptr"], p["indices"]],
                                    [p["full_indptr"], p["full_indices"]], c["full"], c["q"], k,
                                    ef, c["d_p"], gpu_order=True, stages=3)
    assert torch.equal(t_I.cpu(), w_I)
    assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))


def test_ragged_rows_pads_duplicates_and_sparse_handoff(oracle_lib):
    """Rows cut short by -1, a repeated id inside a row, queries whose handoff is
    mostly pads, ids outside the sample: the cases upstream's loops guard against
    (traverse_cpu.cpp:47-49, 109-116)."""
    from pilotann_b200 import extension
    ef, k, B = 32, 10, 64
    c = _case(n=6000, d=64, d_p=32, ef=ef, law="fuzz", batch=B, seed=53)
    p = c["p"]
    n = c["full"].size(0)
    g = torch.Generator().manual_seed(9)
    full_indices = p["full_indices"].clone().reshape(n, 32)
    cut = torch.randint(n, (n // 3,), generator=g)
    full_indices[cut, 20:] = -1                              # rows ending early
    full_indices[cut[:500], 7] = full_indices[cut[:500], 3]  # a repeated id
    full_indices = full_indices.reshape(-1).contiguous()
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), full_indices.cuda(), 32)
    hI = c["hand_I"].reshape(B, -1).clone()
    hD = c["hand_D"].reshape(B, -1).clone()
    hI[:8, 5:] = -1                                          # almost empty handoffs
    hD[:8, 5:] = float("inf")
    hI[8:12] = -1                                            # nothing at all
    pool = extension.VisitedPool(n, 16)
    t_I, t_D = extension.refine(hI, hD, c["q_cuda"], c["full_cuda"], c["nbr"], c["row_of"],
                                full_nbr, pool, ef, c["d_p"], k=k)
    torch.cuda.synchronize()
    w_I, w_D = oracle_lib.refine_ex(hI.cpu().clone(), hD.cpu().clone(),
                                    [p["indptr"], p["indices"]],
                                    [p["full_indptr"], full_indices], c["full"], c["q"], k, ef,
                                    c["d_p"], gpu_order=True, stages=3)
    assert torch.equal(t_I.cpu(), w_I)
    assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))
    assert (t_I[8:12] == -1).all()


def test_rejections():
    from pilotann_b200 import _C
    lib = _C.lib()
    # stages must be 2 or 3
    rc = lib.pa_refine(0, 0, 0, 0, 0, 0, 0, 0, 32, 0, 32, 4, 100, 64, 32, 64, 16, 10, 1, 0, 0, 0)
    assert rc == _C.PA_ERR_ARG and b"stages" in lib.pa_last_error()
    # k larger than the candidate row
    rc = lib.pa_refine(0, 0, 0, 0, 0, 0, 0, 0, 32, 0, 32, 4, 100, 64, 32, 64, 16, 100, 3, 0, 0, 0)
    assert rc == _C.PA_ERR_ARG and b"k must" in lib.pa_last_error()
    # d_principle > d_model
    rc = lib.pa_refine(0, 0, 0, 0, 0, 0, 0, 0, 32, 0, 32, 4, 100, 64, 96, 64, 16, 10, 3, 0, 0, 0)
    assert rc == _C.PA_ERR_ARG
    # a pool for fewer nodes is refused at creation of the call, and n_slots <= 0 at creation
    import ctypes
    h = ctypes.c_void_p()
    assert lib.pa_visited_pool_create(ctypes.byref(h), 100, 0) == _C.PA_ERR_ARG
    assert lib.pa_visited_pool_bytes(1000, 4) == 4 * 1008 + 32


def test_large_ef_and_wide_rows(oracle_lib):
    """ef_search 1024: heaps of 1024 / 2048 entries and a 4096-entry handoff row (more
    shared memory than a CTA gets by default, so the launch opts in), the traversal
    pads the handoff beyond its 256-entry heaps with (-1, -inf); and a degree-64
    sub-graph (two 32-slot chunks per adjacency row)."""
    from pilotann_b200 import extension
    from helpers import make_problem
    k = 10
    for ef, n_nb in ((1024, 32), (64, 64)):
        B, d, d_p = 48, 64, 32
        p = make_problem(n=6000, d=d, n_nb=n_nb, ratio=0.5, batch=B, n_init=32, seed=61)
        full = p["full"]
        reduced = p["storage"][:, :d_p].contiguous()
        q = p["query"]
        g = torch.Generator().manual_seed(3)
        ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 32), generator=g)]
        init_D = ((q[:, :d_p].unsqueeze(1) - full[ids][:, :, :d_p]) ** 2).sum(-1).contiguous()
        nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(),
                                           p["mapping"].cuda(), reduced.size(0), n_nb)
        hI = torch.empty(B, 4, ef, dtype=torch.int64, device="cuda")
        hD = torch.empty(B, 4, ef, device="cuda")
        extension.traverse_packed(hI, hD, nbr, row_of, reduced.cuda(), q[:, :d_p].contiguous().cuda(),
                                  ids.cuda(), init_D.cuda(), n_nb)
        full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), n_nb)
        pool = extension.VisitedPool(full.size(0), 16)
        st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
        t_I, t_D = extension.refine(hI, hD, q.cuda(), full.cuda(), nbr, row_of, full_nbr, pool, ef,
                                    d_p, k=k, stats=st)
        torch.cuda.synchronize()
        w_I, w_D, w_st = oracle_lib.refine_ex(hI.reshape(B, -1).cpu(), hD.reshape(B, -1).cpu(),
                                              [p["indptr"], p["indices"]],
                                              [p["full_indptr"], p["full_indices"]], full, q, k, ef,
                                              d_p, gpu_order=True, with_stats=True)
        assert torch.equal(t_I.cpu(), w_I), (ef, n_nb)
        assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))
        assert torch.equal(st.cpu(), w_st)


def test_shape_sweep_vs_oracle(oracle_lib):
    """Odd shapes: dimensions that are not multiples of 128 (or of 32), d_principle
    anywhere up to d, ef 1 (a 4-entry handoff under 16-entry heaps), heaps that are
    not powers of two, k from 1 to the whole row -- all bit for bit."""
    from pilotann_b200 import extension
    from helpers import make_problem
    g = torch.Generator().manual_seed(77)
    shapes = [(8, 4, 1, 1), (8, 8, 3, 5), (20, 12, 16, 10), (64, 16, 17, 1), (100, 64, 33, 40),
              (132, 128, 100, 25), (256, 64, 300, 50), (36, 36, 40, 160)]
    for d, d_p, ef, k in shapes:
        B = 24
        p = make_problem(n=3000, d=d, ratio=0.5, batch=B, n_init=32, seed=80 + d)
        full, q = p["full"], p["query"]
        ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 4 * ef), generator=g)]
        ids[torch.rand(B, 4 * ef, generator=g) < 0.15] = -1
        dist = ((q[:, :d_p].unsqueeze(1) - full[ids.clamp_min(0)][:, :, :d_p]) ** 2).sum(-1)
        dist[ids < 0] = float("inf")
        dist = dist.contiguous()
        reduced = p["storage"][:, :d_p].contiguous()
        nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(),
                                           p["mapping"].cuda(), reduced.size(0), 32)
        full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
        pool = extension.VisitedPool(full.size(0), 7)
        st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
        t_I, t_D = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of,
                                    full_nbr, pool, ef, d_p, k=k, stats=st)
        torch.cuda.synchronize()
        w_I, w_D, w_st = oracle_lib.refine_ex(ids.clone(), dist.clone(), [p["indptr"], p["indices"]],
                                              [p["full_indptr"], p["full_indices"]], full, q, k, ef,
                                              d_p, gpu_order=True, with_stats=True)
        assert torch.equal(t_I.cpu(), w_I), (d, d_p, ef, k)
        assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32)), (d, d_p, ef, k)
        assert torch.equal(st.cpu(), w_st), (d, d_p, ef, k)


def test_three_warp_ctas_for_short_rows(oracle_lib):
    """Rows of at most 128 floats and more queries than nine per SM: the kernel runs
    with a heap warp and two gather warps (twelve CTAs per SM) instead of three or four.
    Same bits as the oracle, and as the same queries refined in small batches (which
    take the wider CTAs)."""
    from pilotann_b200 import extension
    from helpers import make_problem
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B, d, d_p, ef, k = 9 * sms + 170, 64, 32, 24, 10
    g = torch.Generator().manual_seed(5)
    p = make_problem(n=3000, d=d, ratio=0.5, batch=B, n_init=32, seed=91)
    full, q = p["full"], p["query"]
    ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 4 * ef), generator=g)]
    dist = ((q[:, :d_p].unsqueeze(1) - full[ids][:, :, :d_p]) ** 2).sum(-1).contiguous()
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
    assert extension.refine_wave(d) == 12 * sms and extension.refine_wave(768) == 7 * sms
    pool = extension.VisitedPool(full.size(0), B)
    st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
    args = (full.cuda(), nbr, row_of, full_nbr, pool, ef, d_p)
    t_I, t_D = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), *args, k=k, stats=st)
    torch.cuda.synchronize()
    w_I, w_D, w_st = oracle_lib.refine_ex(ids.clone(), dist.clone(), [p["indptr"], p["indices"]],
                                          [p["full_indptr"], p["full_indices"]], full, q, k, ef,
                                          d_p, gpu_order=True, with_stats=True)
    assert torch.equal(t_I.cpu(), w_I)
    assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))
    assert torch.equal(st.cpu(), w_st)
    s_I, s_D = extension.refine(ids[:200].cuda(), dist[:200].cuda(), q[:200].cuda(), *args, k=k)
    assert torch.equal(s_I, t_I[:200]) and torch.equal(s_D.view(torch.int32), t_D[:200].view(torch.int32))


def test_equal_distances_take_upstreams_sequence(oracle_lib):
    """Vectors on a coarse grid, many of them identical: equal distances everywhere.
    The shortcuts of the kernel (two-expansion stage without the open heap, seeds
    merged by selection and sort) give way to upstream's heap sequence wherever two
    keys that matter are equal -- same bits as the oracle, statistics included."""
    from pilotann_b200 import extension
    from helpers import make_problem
    g = torch.Generator().manual_seed(123)
    for d, d_p, ef, k, levels, dup in [(64, 32, 24, 10, 2.0, 6), (96, 32, 48, 10, 1.0, 3),
                                       (200, 64, 16, 5, 4.0, 10), (768, 128, 32, 10, 1.0, 4)]:
        B = 48
        p = make_problem(n=3000, d=d, ratio=0.5, batch=B, n_init=32, seed=300 + d)
        full = torch.round(p["full"] * levels) / levels
        full[torch.randperm(3000, generator=g)] = full.repeat_interleave(dup, 0)[:3000]
        full = full.contiguous()
        q = (torch.round(p["query"] * levels) / levels).contiguous()
        ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 4 * ef), generator=g)]
        ids[torch.rand(B, 4 * ef, generator=g) < 0.1] = -1
        dist = ((q[:, :d_p].unsqueeze(1) - full[ids.clamp_min(0)][:, :, :d_p]) ** 2).sum(-1)
        dist[ids < 0] = float("inf")
        dist = dist.contiguous()
        nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                           p["storage"].size(0), 32)
        full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
        pool = extension.VisitedPool(full.size(0), 16)
        graphs = ([p["indptr"], p["indices"]], [p["full_indptr"], p["full_indices"]])
        for stages_k in (None, k):
            st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
            t_I, t_D = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of,
                                        full_nbr if stages_k else None, pool, ef, d_p, k=stages_k,
                                        stats=st)
            torch.cuda.synchronize()
            w_bI, w_bD = ids.clone(), dist.clone()
            w_I, w_D, w_st = oracle_lib.refine_ex(w_bI, w_bD, *graphs, full, q, k, ef, d_p, gpu_order=True,
                                                  stages=3 if stages_k else 2, with_stats=True)
            if stages_k is None:
                w_I, w_D, w_st = w_bI, w_bD, w_st[:, :2]
                st = st[:, :2]
            assert torch.equal(t_I.cpu(), w_I), (d, ef, stages_k)
            assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32)), (d, ef, stages_k)
            assert torch.equal(st.cpu(), w_st), (d, ef, stages_k)
        # the case is what it claims to be: equal distances among a query's candidates
        row = dist[0][ids[0] >= 0]
        assert row.unique().numel() < row.numel()


@pytest.mark.parametrize("ef,k,spoil", [(16, 16, None), (30, 10, "pairs"), (48, 48, "pairs"),
                                        (64, 10, "nan"), (96, 90, "pairs"), (128, 100, "pairs"),
                                        (150, 10, "nan"), (192, 100, "pairs"), (256, 200, "pairs"),
                                        (257, 20, "pairs")])
def test_result_list_of_every_capacity(oracle_lib, ef, k, spoil):
    """Every capacity of the result list in registers (16 .. 256, the next one has the
    array heaps), with long results; "pairs": some vectors twice, so that a few equal
    distances reach the merges and the log of admissions is replayed; "nan": a vector
    of NaN that searches meet, which sends the query back to the array heaps.  Bit for
    bit the oracle's, statistics included (with NaN, which the heaps do not order, for the
    queries that do not meet one)."""
    from pilotann_b200 import extension
    from helpers import make_problem
    B, n, d, d_p = 40, 4000, 48, 16
    g = torch.Generator().manual_seed(1000 + ef)
    p = make_problem(n=n, d=d, ratio=0.5, batch=B, n_init=32, seed=700)
    full, q = p["full"].clone(), p["query"]
    if spoil == "pairs":
        twins = torch.randperm(n, generator=g)[:400].view(2, -1)
        full[twins[0]] = full[twins[1]]
    ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 4 * ef), generator=g)]
    if spoil == "nan":
        # a neighbour of the first candidates, itself no candidate
        bad = p["full_indices"][p["full_indptr"][ids[::8, 0]]].unique()
        full[bad] = float("nan")
        keep = ids[~torch.isin(ids, bad)]
        ids = keep[torch.randint(keep.numel(), (B, 4 * ef), generator=g)]
    dist = ((q[:, :d_p].unsqueeze(1) - full[ids][:, :, :d_p]) ** 2).sum(-1).contiguous()
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
    pool = extension.VisitedPool(n, 16)
    graphs = ([p["indptr"], p["indices"]], [p["full_indptr"], p["full_indices"]])
    for top in (None, k):
        st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
        t_I, t_D = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of,
                                    full_nbr, pool, ef, d_p, k=top, stats=st)
        torch.cuda.synchronize()
        w_bI, w_bD = ids.clone(), dist.clone()
        w_I, w_D, w_st = oracle_lib.refine_ex(w_bI, w_bD, *graphs, full, q, k, ef, d_p, gpu_order=True,
                                              stages=3 if top else 2, with_stats=True)
        if top is None:
            w_I, w_D, w_st, st = w_bI, w_bD, w_st[:, :2], st[:, :2]
        if spoil == "nan":
            same = (t_I.cpu() == w_I).all(1) & (t_D.cpu() == w_D).all(1) & (st.cpu() == w_st).all(1)
            assert ((t_I >= -1) & (t_I < n)).all()
            if top is None:                      # (the full-graph stage meets one always)
                assert 0.2 < same.float().mean() < 1.0
            else:
                exact = (q.unsqueeze(1) - full[t_I.cpu()]).square().sum(-1)
                assert torch.allclose(t_D.cpu(), exact, rtol=1e-4, atol=1e-6)
            again = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of,
                                     full_nbr, pool, ef, d_p, k=top)
            assert torch.equal(again[0], t_I)
            continue
        assert torch.equal(t_I.cpu(), w_I), top
        assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32)), top
        assert torch.equal(st.cpu(), w_st), top


@pytest.mark.parametrize("per_sm,d,ef", [(2, 48, 24), (2, 768, 40), (4, 768, 128), (4, 48, 256),
                                         (2, 2048, 64)])
def test_ctas_for_few_queries_per_sm(oracle_lib, per_sm, d, ef):
    """Two and four queries per SM: CTAs of 16 and 8 warps, with long rows and short ones.
    Bit for bit the oracle's."""
    from pilotann_b200 import extension
    from helpers import make_problem
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    base, n, d_p, k = 24, 6000, 16, 10
    g = torch.Generator().manual_seed(d + ef)
    p = make_problem(n=n, d=d, ratio=0.5, batch=base, n_init=32, seed=800, exact_entries=False)
    full, q = p["full"], p["query"]
    ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (base, 4 * ef), generator=g)]
    dist = ((q[:, :d_p].unsqueeze(1) - full[ids][:, :, :d_p]) ** 2).sum(-1).contiguous()
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
    w_I, w_D, w_st = oracle_lib.refine_ex(ids.clone(), dist.clone(), [p["indptr"], p["indices"]],
                                          [p["full_indptr"], p["full_indices"]], full, q, k, ef,
                                          d_p, gpu_order=True, with_stats=True)
    times = per_sm * sms // base
    B = times * base
    pool = extension.VisitedPool(n, B)
    st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
    for _ in range(2):                                     # the second launch finds used slots
        t_I, t_D = extension.refine(ids.repeat(times, 1).cuda(), dist.repeat(times, 1).cuda(),
                                    q.repeat(times, 1).cuda(), full.cuda(), nbr, row_of, full_nbr,
                                    pool, ef, d_p, k=k, stats=st)
        torch.cuda.synchronize()
        assert torch.equal(t_I.cpu(), w_I.repeat(times, 1))
        assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32).repeat(times, 1))
        assert torch.equal(st.cpu(), w_st.repeat(times, 1))


@pytest.mark.parametrize("d,d_p", [(36, 4), (36, 12), (36, 32), (68, 4), (100, 36), (104, 36)])
def test_short_residuals(oracle_lib, d, d_p):
    """Seeds completed over at most 32 and 64 trailing dimensions share a warp by four and
    by two; one more group of four dimensions takes the whole warp."""
    from pilotann_b200 import extension
    from helpers import make_problem
    B, n, ef = 16, 3000, 37
    g = torch.Generator().manual_seed(d * 100 + d_p)
    p = make_problem(n=n, d=d, ratio=0.5, batch=B, n_init=32, seed=900 + d)
    full, q = p["full"], p["query"]
    ids = p["nodelist"][torch.randint(p["nodelist"].numel(), (B, 4 * ef), generator=g)]
    ids[torch.rand(B, 4 * ef, generator=g) < 0.2] = -1
    dist = ((q[:, :d_p].unsqueeze(1) - full[ids.clamp_min(0)][:, :, :d_p]) ** 2).sum(-1)
    dist[ids < 0] = float("inf")
    dist = dist.contiguous()
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    pool = extension.VisitedPool(n, B)
    t_I, t_D = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of, None,
                                pool, ef, d_p)
    torch.cuda.synchronize()
    w_I, w_D = ids.clone(), dist.clone()
    oracle_lib.refine_ex(w_I, w_D, [p["indptr"], p["indices"]],
                         [p["full_indptr"], p["full_indices"]], full, q, 10, ef, d_p,
                         gpu_order=True, stages=2)
    assert torch.equal(t_I.cpu(), w_I)
    assert torch.equal(t_D.cpu().view(torch.int32), w_D.view(torch.int32))


def _on_array_heaps(ids, dist, q, full, sub, graph, k, ef, H, d_p):
    """The refinement of one query with upstream's array heaps in the comparisons of the
    kernel's (they differ from the oracle's for NaN only), the node it prepares ahead
    included: with NaN in the open heap that is not always the one popped next, and its
    neighbours stay marked.  Returns what both stages leave, expansions and evaluations, and
    the most results a stage admitted."""
    inf = float("inf")

    def sink(h, me):
        n, c = len(h), 0
        while 2 * c + 1 < n:
            child = 2 * c + 1
            if child + 1 < n and h[child + 1][0] < h[child][0]:
                child += 1
            if not h[child][0] < me[0]:
                break
            h[c], c = h[child], child
        h[c] = me

    def pop(h):
        out = h[0]
        sink(h, (inf, -1))
        return out

    def pushpop(h, key, v):
        if not key <= h[0][0]:
            sink(h, (key, v))

    def replace(h, key, v):
        n, c = len(h), 0
        while 2 * c + 1 < n:
            child = 2 * c + 1
            if child + 1 < n and h[child + 1][0] > h[child][0]:
                child += 1
            c = child
        if key >= h[c][0]:
            return
        while c > 0 and h[(c - 1) // 2][0] > key:
            h[c], c = h[(c - 1) // 2], (c - 1) // 2
        h[c] = (key, v)

    visited, stats, admitted = set(), [], 0

    def stage(seeds, csr, max_iter, k_out, ahead):
        nonlocal admitted
        res, open_ = [(-inf, -1)] * H, [(inf, -1)] * (2 * H)
        for v, key in seeds:
            if v >= 0:
                visited.add(v)
                replace(open_, key, v)

        def gather(u):
            row = [v for v in csr[1][csr[0][u]:csr[0][u + 1]].tolist() if v not in visited]
            visited.update(row)
            return [(((q - full[v]) ** 2).sum().item(), v) for v in row]

        n_expand = n_eval = n_push = 0
        key, u = pop(open_)
        guess = None
        for step in range(max_iter):
            if u < 0 or key >= -res[0][0]:
                break
            if guess is None or guess[0] != u:
                guess = (u, gather(u))
            new, root = guess[1], open_[0]
            n_expand += 1
            n_eval += len(new)
            for dv, v in new:
                if not dv >= -res[0][0]:
                    pushpop(res, -dv, v)
                    replace(open_, dv, v)
                    n_push += 1
            guess = None
            if step + 1 < max_iter:
                if ahead:
                    best = min((x for x in new if x[0] < inf), key=lambda x: x[0], default=(inf, -1))
                    at = best[1] if best[0] < root[0] else root[1]
                    guess = (at, gather(at)) if at >= 0 else None
                key, u = pop(open_)
        admitted = max(admitted, n_push)
        stats.extend((n_expand, n_eval))
        for v, key in seeds:
            if v >= 0:
                pushpop(res, -key, v)
        for _ in range(k_out, H):
            pop(res)
        out = [pop(res) for _ in range(k_out)][::-1]
        return [(v, -key) for key, v in out]

    seeds = [(v, dv + ((q[d_p:] - full[v][d_p:]) ** 2).sum().item() if v >= 0 else dv)
             for v, dv in zip(ids.tolist(), dist.tolist())]
    first = stage(seeds, sub, min(2, 2 * ef), len(seeds), False)
    last = stage(first, graph, min(1024, 2 * ef), k, True)
    return first, last, stats, admitted


@pytest.mark.parametrize("ef,k,n_cand,spoil", [
    (48, 10, 192, "seed distance"), (96, 20, 384, "seed distance"), (192, 10, 768, "seed distance"),
    (64, 10, 256, "seed vector"), (128, 60, 512, "seed vector"), (256, 10, 1024, "seed vector"),
    (30, 10, 120, "neighbour"), (100, 10, 400, "neighbour"), (150, 30, 600, "neighbour"),
    (257, 10, 1028, "seed distance"), (257, 10, 1028, "seed vector"), (257, 10, 1028, "neighbour"),
    (48, 40, 40, "twins"), (100, 60, 60, "twins"), (192, 90, 92, "twins"), (257, 60, 60, "twins"),
    (48, 10, 40, "unsampled twins"), (100, 10, 60, "unsampled twins"),
    (192, 10, 92, "unsampled twins")])
def test_queries_sent_back_to_the_array_heaps(ef, k, n_cand, spoil):
    """What makes a query leave the result list for the array heaps, for each width of the
    list and for the heaps alone (ef 257): a NaN among the seeds, in the distance that came
    with it or in its vector, a NaN among the neighbours, equal distances in the sub-graph
    stage, and equal distances met only in the full-graph stage after more admissions than the
    log holds (few candidates: H of them).  Vectors on a grid, so
    that every distance is exact in any order of additions; rows, distances and statistics are
    those of the array heaps, and two runs agree."""
    from pilotann_b200 import extension
    B, n, d, d_p = 12, 3000, 48, 16
    g = torch.Generator().manual_seed(ef + n_cand)
    p = make_problem(n=n, d=d, ratio=0.5, batch=B, n_init=32, seed=700)
    full, q = (torch.round(p[x] * 128) / 128 for x in ("full", "query"))
    if spoil.endswith("twins"):
        at = torch.randperm(n, generator=g)
        if spoil == "unsampled twins":
            at = at[~torch.isin(at, p["nodelist"])]
        at = at[:at.numel() // 2 * 2].view(2, -1)
        full[at[0]] = full[at[1]]
    ids = torch.stack([p["nodelist"][torch.randperm(p["nodelist"].numel(), generator=g)[:n_cand]]
                       for _ in range(B)])
    dist = ((q[:, :d_p].unsqueeze(1) - full[ids][:, :, :d_p]) ** 2).sum(-1)
    hit = torch.arange(B) % 3 == 0                  # (the others may stay clean)
    if spoil == "seed distance":
        dist[hit, 5] = dist[hit, n_cand // 2] = float("nan")
    elif spoil == "seed vector":
        full[ids[hit][:, [3, n_cand - 1]].reshape(-1), d_p:] = float("nan")
    elif spoil == "neighbour":
        best = ids[hit].gather(1, dist[hit].argmin(1, keepdim=True)).reshape(-1)
        bad = p["full_indices"].view(n, -1)[best, :2].reshape(-1)
        full[bad] = float("nan")
        dist[torch.isin(ids, bad)] = float("nan")
    dist = dist.contiguous()
    H = extension.cpu_heap_size_for(ef)
    csr = [[p[a].contiguous(), p[b]] for a, b in (("indptr", "indices"), ("full_indptr", "full_indices"))]
    want = [_on_array_heaps(ids[b], dist[b], q[b].double(), full.double(), *csr, k, ef, H, d_p)
            for b in range(B)]
    if spoil.endswith("twins"):                     # the case is what it claims to be
        early, late = ([any(a[1] == b[1] and a[0] >= 0 for a, b in zip(w[i], w[i][1:max(k, 26) + 1]))
                        for w in want] for i in (0, 1))
        if spoil == "twins":
            assert any(early)
        else:
            assert any(y and not x and w[3] > H for w, x, y in zip(want, early, late))
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
    pool = extension.VisitedPool(n, 16)
    for stage, top in ((0, None), (1, k)):
        runs = []
        for _ in range(2):
            st = torch.zeros(B, 4, dtype=torch.int32, device="cuda")
            got = extension.refine(ids.cuda(), dist.cuda(), q.cuda(), full.cuda(), nbr, row_of,
                                   full_nbr, pool, ef, d_p, k=top, stats=st)
            torch.cuda.synchronize()
            runs.append([got[0].cpu(), got[1].cpu(), st.cpu()])
        for x, y in zip(*runs):
            assert torch.equal(x.nan_to_num(-7), y.nan_to_num(-7)) if x.is_floating_point() else torch.equal(x, y)
        w_I = torch.tensor([[v for v, _ in w[stage]] for w in want])
        w_D = torch.tensor([[dv for _, dv in w[stage]] for w in want])
        w_st = torch.tensor([w[2] for w in want], dtype=torch.int32)
        got_I, got_D, st = runs[0]
        wrong = (got_I != w_I).any(1).nonzero().flatten().tolist()
        assert not wrong, (top, wrong)
        assert torch.equal(got_D.nan_to_num(-7, 1e30, -1e30), w_D.nan_to_num(-7, 1e30, -1e30)), top
        assert torch.equal(st[:, :2 + 2 * stage], w_st[:, :2 + 2 * stage]), top


@pytest.mark.skipif("PA_REFINE_PROFILE=1" not in os.environ.get("PILOTANN_B200_DEFINES", ""),
                    reason="needs a library built with PILOTANN_B200_DEFINES=PA_REFINE_PROFILE=1")
@pytest.mark.parametrize("ef", [48, 257])
def test_phases_of_a_profile_build(ef):
    """What a profile build counts per query: the heap warp's phases (set-up, seed inserts, pops,
    waiting, inserts, merge, then pushes in units), the gather warp's.  All of them are
    there and either side's clocks add up to the same time; the result list in registers (ef 48) and the array heaps (ef 257)."""
    from pilotann_b200 import extension
    c = _case(n=4000, batch=64, ef=ef)
    pool = extension.VisitedPool(c["full"].size(0), 64)
    st = torch.zeros(64, 24, dtype=torch.int32, device="cuda")
    extension.refine(c["hand_I"], c["hand_D"], c["q_cuda"], c["full_cuda"], c["nbr"], c["row_of"],
                     c["full_nbr"], pool, ef, c["d_p"], k=10, stats=st)
    heap, gather = st[:, 4:12].cpu().long(), st[:, 12:].cpu().long()
    assert (st[:, 2] > 1).all()
    assert (heap.sum(0) > 0).all(), heap.sum(0)
    assert (gather[:, [0, 1, 2, 4, 5, 6, 7, 8]].sum(0) > 0).all(), gather.sum(0)   # (3: long rows)
    whole = heap[:, :7].sum(1).double() / gather.sum(1).double()
    assert (whole > 0.8).all() and (whole < 1.25).all()


def test_replay_of_upstream_fixtures():
    """Outputs of upstream ``traverse_refine`` recorded by tests/golden/make_golden.py
    (CPU, no GPU involved), replayed through the refinement kernel without the
    upstream module: top-k, and the handoff rows the sub-graph stage leaves."""
    from pathlib import Path
    from pilotann_b200 import extension
    gold = torch.load(Path(__file__).parent / "golden" / "golden_cpu.pt")
    p = gold["problem"]
    n = p["full"].size(0)
    d_sub = p["storage"].size(1)
    nbr, row_of = extension.pack_graph(p["indptr"].cuda(), p["indices"].cuda(), p["mapping"].cuda(),
                                       p["storage"].size(0), 32)
    full_nbr = extension.pack_fullgraph(p["full_indptr"].cuda(), p["full_indices"].cuda(), 32)
    pool = extension.VisitedPool(n, 8)
    assert d_sub == p["full"].size(1)
    for ef, fx in gold["refine"].items():
        k = fx["out_I"].size(1)
        args = (fx["cand_I"].cuda(), fx["cand_D"].cuda(), p["query"].cuda(), p["full"].cuda(), nbr,
                row_of)
        t_I, t_D = extension.refine(*args, full_nbr, pool, ef, fx["d_principle"], k=k)
        s_I, s_D = extension.refine(*args, None, pool, ef, fx["d_principle"], k=None)
        torch.cuda.synchronize()
        assert (t_I.cpu() == fx["out_I"]).float().mean().item() >= 0.995, ef
        assert torch.allclose(t_D.cpu(), fx["out_D"], rtol=1e-5, atol=1e-6)
        assert (s_I.cpu() == fx["buffer_I"]).float().mean().item() >= 0.995
        fin = torch.isfinite(fx["buffer_D"])
        assert torch.equal(fin, torch.isfinite(s_D.cpu()))
        assert torch.allclose(s_D.cpu()[fin], fx["buffer_D"][fin], rtol=1e-5, atol=1e-6)
