"""Kernel and dispatch edges: the sizes where a tile, a remainder or a choice of variant can go wrong, against the
CPU oracle (or float64 where the oracle has no such op)."""
import numpy as np
import pytest
import torch

from deers_b200 import _lib
from tests.helpers import TOL_F16, assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,T", [(8, 1), (56, 129), (72, 127), (80, 300), (120, 257)])
def test_f16_head_dims_in_place_with_strided_rows(D, T):
    """Head dims between the tile widths: the columns a tile has beyond head_dim must neither be read (they belong to
    the neighbouring head of a [B,T,3C] buffer here) nor written (the output is a slice of a larger buffer)."""
    from deers_b200 import ops
    from oracle import ref
    B, H = 2, 3
    C = H * D
    rng = np.random.default_rng(D + T)
    qkv = torch.from_numpy(rng.standard_normal((B, T, 3 * C)).astype(np.float16)).cuda()
    q, k, v = (qkv[..., i * C:(i + 1) * C].view(B, T, H, D).permute(0, 2, 1, 3) for i in range(3))
    do = torch.from_numpy(rng.standard_normal((B, H, T, D)).astype(np.float16)).cuda()
    big = torch.full((B, T, H, D + 8), 7.0, dtype=torch.float16, device="cuda")
    out = big[..., :D].permute(0, 2, 1, 3)
    scale = ops.default_scale(D)
    o, lse = ops.attention_fwd(q, k, v, scale, out=out)
    dvb = torch.full((B, T, H, D + 8), 7.0, dtype=torch.float16, device="cuda")
    for ws_pass in (1, 2):
        ws = torch.empty(ops.workspace_bytes(q, scale, True, ws_pass), dtype=torch.uint8, device="cuda")
        dq, dk, dv = ops.attention_bwd(q, k, v, o, lse, do, scale, workspace=ws, dv_out=dvb[..., :D].permute(0, 2, 1, 3))
        ops.Context.current(q.device).sync()
        host = [t.float().cpu().numpy() for t in (q, k, v, do)]
        want = ref.attn_fwd_bwd(*[np.ascontiguousarray(a) for a in host])
        for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), (o, lse, dq, dk, dv), want):
            assert_close(g.float().cpu().numpy(), w, TOL_F16, f"D {D} T {T} {name}")
    assert torch.all(big[..., D:] == 7.0) and torch.all(dvb[..., D:] == 7.0), "columns beyond head_dim are not ours"


@pytest.mark.parametrize("M,N,K", [(1, 3, 5), (31, 33, 63), (32, 32, 64), (33, 65, 65), (63, 129, 191), (64, 64, 1025),
                                   (100, 40, 4099), (192, 190, 1023), (1024, 576, 70), (2050, 1030, 40)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 1), (0, 0), (1, 1), (1, 0)])
@pytest.mark.parametrize("aligned", [True, False])
def test_f32_gemm_tiles_clusters_and_remainders(M, N, K, a_mn, b_mn, aligned):
    """Every tile variant, K split over a cluster or not, with tiles, stages and parts that do not come out even."""
    from deers_b200 import gpt
    rng = np.random.default_rng(M + 7 * N + 13 * K)
    a = rng.standard_normal((M, K)).astype(np.float32)
    b = rng.standard_normal((K, N)).astype(np.float32)
    want = a.astype(np.float64) @ b.astype(np.float64)

    def place(x):
        pad = 0 if aligned else 3                          # an odd leading dimension rules out 16-byte copies
        big = torch.full((x.shape[0], x.shape[1] + pad), float("nan"), device="cuda")
        big[:, :x.shape[1]] = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        return big[:, :x.shape[1]]
    ta, tb = place(a.T if a_mn else a), place(b if b_mn else b.T)
    big = torch.full((M + 1, N + 3), float("nan"), device="cuda")
    got = gpt.gemm_f32(ta, tb, bool(a_mn), bool(b_mn), out=big[:M, :N])
    torch.cuda.synchronize()
    # K rounded sums of unit-variance products: sqrt(K) growth, 2^-24 each, against sqrt(K) * (largest of the draws)
    tol = 2e-6 * max(1.0, np.sqrt(K) / 4) * max(1.0, np.abs(want).max())
    assert np.abs(got.cpu().numpy() - want).max() <= tol
    assert torch.isnan(big[M]).all() and torch.isnan(big[:M, N:]).all(), "nothing outside C is written"


@pytest.mark.parametrize("T", [1, 31, 33, 64, 129, 257])
@pytest.mark.parametrize("D", [3, 32, 36, 64, 92, 96, 100, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_f32_attention_tiles_and_groups(T, D, causal):
    """Rows per block, tiles per group and head-dim paddings that do not come out even; D = 3 takes the element path."""
    from deers_b200 import ops
    from oracle import ref
    from tests.helpers import TOL_F32
    rng = np.random.default_rng(T * 131 + D)
    host = [rng.standard_normal((2, 2, T, D)).astype(np.float32) for _ in range(4)]
    q, k, v, do = (torch.from_numpy(a).cuda() for a in host)
    op = ops.CausalAttention.new(q, k, v, None, causal)
    o = op.forward()
    grads = ops.GradientStore()
    op.backward(grads, do)
    ops.Context.current(q.device).sync()
    want = ref.attn_fwd_bwd(*host, causal=causal)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), [o, op.lse] + [grads.get(t) for t in (q, k, v)], want):
        g = g.cpu().numpy()
        if T == 1 and name in ("dq", "dk"):
            # P = 1, so dS = dP - delta cancels to zero; what is left is the rounding of two D-term sums of dO * V,
            # each within D * 2^-24 * sum |dO V|, times scale and the other operand (the oracle's own is as large)
            sums = np.abs(host[3] * host[2]).sum(-1).max()
            other = np.abs(host[1] if name == "dq" else host[0]).max()
            assert np.abs(g - w).max() <= 4 * D * 2.0 ** -24 * sums * D ** -0.5 * other, name
        else:
            assert_close(g, w, TOL_F32, f"T {T} D {D} {name}")


def test_gpt_forward_lengths_share_graphs_and_follow_the_weights():
    """Every length must give what the oracle gives, in whatever order lengths come,
    before and after an optimizer step and after a weight upload (the head's f16 pair is kept between calls)."""
    from deers_b200 import gpt
    from oracle import ref
    V, L, H, C, Hm, Tmax, B = 1030, 2, 2, 64, 128, 70, 2
    cfg = (V, L, H, C, Hm)
    params = ref.gpt_init_params(cfg, seed=3)
    m = gpt.GPT(gpt.GPTConfig(V, Tmax, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    m.load_parameters(params)
    rng = np.random.default_rng(4)
    ids = rng.integers(0, V, (B, Tmax))

    def check(T, b=B):
        got = m.forward(torch.from_numpy(ids[:b, :T].copy()).cuda())
        m.ctx.sync()
        want = ref.gpt_step(cfg, params, ids[:b, :T], want_grads=False)["logits"]
        # f32 sums of up to 1030 terms through two layers against the oracle's left-to-right sums
        assert_close(got.cpu().numpy().reshape(np.asarray(want).shape), want, 1e-4, f"T {T}")
    for T in (31, 32, 30, 33, 1, 33, 64, 40, 65, 70, 66, 69, 31, 5):
        check(T)
    check(50, 1), check(51, 1), check(52, 1)
    tgt = torch.from_numpy(rng.integers(0, V, (B, 20))).cuda()
    m.train_step(torch.from_numpy(ids[:, :20].copy()).cuda(), tgt, lr=1e-2)
    m.ctx.sync()
    params = [m.parameter(i) for i in range(m.num_parameters())]
    check(40), check(41)
    params = ref.gpt_init_params(cfg, seed=5)
    m.load_parameters(params)
    check(42), check(31)


@pytest.mark.parametrize("B,H,T,D,causal", [(4, 100, 100, 64, True), (3, 133, 60, 128, True), (2, 149, 129, 64, True), (1, 200, 385, 128, True),
                                            (5, 60, 250, 128, False), (1, 3, 1025, 64, False)])
def test_f16_attention_short_items_in_a_row(B, H, T, D, causal):
    """Every SM walks several items of one, two, three ... key tiles: items without a step of one softmax group, odd and even
    step counts, the deferred epilogues.  Keys grow along the sequence, so the reference maximum moves by more than 2^8
    and O is rescaled by either group."""
    from deers_b200 import ops
    from oracle import ref
    rng = np.random.default_rng(T)
    host = [rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4)]
    host[1] *= (1.0 + 3.0 * (np.arange(T) // 128))[None, None, :, None]
    host = [a.astype(np.float16).astype(np.float32) for a in host]
    q, k, v, do = (torch.from_numpy(a).to("cuda", torch.float16) for a in host)
    scale = ops.default_scale(D)
    o, lse = ops.attention_fwd(q, k, v, scale, causal)
    grads = [ops.attention_bwd(q, k, v, o, lse, do, scale, causal, workspace=torch.empty(ops.workspace_bytes(q, scale, causal, p),
                                                                                         dtype=torch.uint8, device="cuda")) for p in (1, 2)]
    ops.Context.current(q.device).sync()
    want = ref.attn_fwd_bwd(*host, causal=causal)
    for got in grads:
        for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), (o, lse) + tuple(got), want):
            assert_close(g.float().cpu().numpy(), w, TOL_F16, name)


@pytest.mark.parametrize("B,H,Tq,Tk,D", [(1, 2, 1, 64, 64), (1, 2, 1, 65, 80), (1, 3, 2, 513, 96), (2, 1, 5, 4096, 32), (1, 1, 3, 4097, 80),
                                         (1, 2, 1, 20001, 128), (1, 2, 7, 7, 48), (60, 12, 1, 130, 72), (1, 1, 9, 300, 256), (75, 8, 3, 50, 24)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_decode_chunks_clusters_and_row_lengths(B, H, Tq, Tk, D, dtype):
    """One chunk, a cluster of chunks, chunks merged by a second launch; rows of any number of 16-byte pieces; chunks that a
    causal query does not see."""
    from deers_b200 import ops
    from oracle import ref
    from tests.helpers import TOL_F32
    rng = np.random.default_rng(Tk + D)
    q, k, v = (rng.standard_normal((B, H, t, D)).astype(np.float32) for t in (Tq, Tk, Tk))
    if dtype == torch.float16:
        q, k, v = (a.astype(np.float16).astype(np.float32) for a in (q, k, v))
    tq, tk, tv = (torch.from_numpy(a).to("cuda", dtype) for a in (q, k, v))
    for causal in (True, False):
        want_o, want_lse = ref.attn_decode(q, k, v, None, causal)
        o, lse = ops.attention_decode(tq, tk, tv, causal=causal, want_lse=True)
        ops.Context.current(tq.device).sync()
        tol = TOL_F16 if dtype == torch.float16 else TOL_F32
        assert_close(o.float().cpu().numpy(), want_o, tol, "o")
        assert_close(lse.cpu().numpy(), want_lse, tol, "lse")


@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (128, 256, 512), (136, 200, 520), (768, 768, 8192), (120, 184, 8200), (1024, 776, 768),
                                   (2000, 2312, 72), (264, 1040, 2056), (128, 8, 1288)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_f16_gemm_split_k_and_tile_widths(M, N, K, a_mn, b_mn):
    """One tile per cluster with its K shared out (parts of unequal length), 192- and 256-wide tiles, ragged edges.  Small
    integers: every sum is exact in f32 and f16, so any K range dropped or counted twice shows."""
    from deers_b200 import ops
    rng = np.random.default_rng(M + N + K)
    a = rng.integers(-1, 2, (K, M) if a_mn else (M, K)).astype(np.float16)
    b = rng.integers(-1, 2, (K, N) if b_mn else (N, K)).astype(np.float16)
    got = ops._gemm(M, N, K, torch.from_numpy(a).cuda(), int(a_mn), torch.from_numpy(b).cuda(), int(b_mn))
    ops.Context.current(got.device).sync()
    af, bf = a.astype(np.float64), b.astype(np.float64)
    want = (af.T if a_mn else af) @ (bf if b_mn else bf.T)
    assert np.abs(want).max() <= 2048
    assert np.array_equal(got.float().cpu().numpy(), want.astype(np.float32))


@pytest.mark.parametrize("B,H,T,D,dtype", [(1, 2, 64, 64, torch.float16), (2, 3, 127, 80, torch.float16), (1, 12, 128, 32, torch.float32)])
def test_chained_kernels_see_their_predecessors(B, H, T, D, dtype):
    """Each kernel of a sequence reads what the one before it (or a copy) has just written, over the same buffers again and
    again: eagerly, and captured with a copy, a kernel and a join of two streams as the predecessor.  Bit for bit the same."""
    from deers_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T)
    src = [torch.randn((B, H, T, D), device="cuda", generator=gen).to(dtype) for _ in range(4)]
    scale = ops.default_scale(D)
    side = torch.cuda.Stream()

    def chain(wait):
        x, out = src[0].clone(), []
        for _ in range(3):
            o, lse = ops.attention_fwd(x, src[1], src[2], scale)
            wait()
            dq, dk, dv = ops.attention_bwd(x, src[1], src[2], o, lse, src[3], scale)
            wait()
            y = ops.attention_decode(dq, dk, o, scale)
            x.copy_(y)                                                  # a copy as the predecessor
            other = torch.cuda.current_stream()
            side.wait_stream(other)
            with torch.cuda.stream(side):
                z = dv + x
            x = ops.attention_decode(y, src[1], src[2], scale)
            wait()
            other.wait_stream(side)                                     # two predecessors
            x = ops.attention_decode(x, z, dv, scale)
            out += [o, lse, dq, dk, dv, y, z, x]
        return out

    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        want = chain(st.synchronize)
        got = [chain(lambda: None) for _ in range(3)]
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            captured = chain(lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for g in got + [captured]:
        for a, b in zip(g, want):
            assert torch.equal(a, b)


def gpt_run(tc_head):
    """Forwards of several lengths, a backward and three optimizer steps of a small model, launched kernel by kernel."""
    from deers_b200 import gpt
    from oracle import ref
    V, L, H, C, Hm, T, B = (1100 if tc_head else 300), 2, 2, 64, 128, 70, 2
    m = gpt.GPT(gpt.GPTConfig(V, T, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    m.load_parameters(ref.gpt_init_params((V, L, H, C, Hm), seed=11))
    m.set_graph(False)
    rng = np.random.default_rng(12)
    ids, tgt = (torch.from_numpy(rng.integers(0, V, (B, T))).cuda() for _ in range(2))
    out = [m.forward(ids[:, :t].contiguous()) for t in (1, 33, 64, 70)]
    out.append(m.forward_backward(ids, tgt))
    for _ in range(3):
        out += list(m.train_step(ids, tgt, lr=1e-2, weight_decay=0.1, max_grad_norm=1.0))
        out.append(m.forward(ids))
    m.ctx.sync()
    return [t.cpu().numpy() for t in out] + [m.parameter(i) for i in range(m.num_parameters())] + [m.grad(i) for i in range(m.num_parameters())]


@pytest.mark.parametrize("tc_head", [True, False])
def test_chained_gpt_kernels_see_their_predecessors(tc_head, tmp_path):
    """The kernels of a model's forward, backward and optimizer step, each started while the one before it ends, give bit for
    bit what they give in a process where every launch is waited for."""
    import os
    import subprocess
    import sys
    path = str(tmp_path / "want.npz")
    code = f"import numpy as np; from tests.test_edges_gpu import gpt_run; np.savez({path!r}, *gpt_run({tc_head}))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, cwd=root, timeout=300, env=dict(os.environ, CUDA_LAUNCH_BLOCKING="1"))
    want = np.load(path)
    for _ in range(3):
        got = gpt_run(tc_head)
        assert len(got) == len(want.files)
        for i, g in enumerate(got):
            assert np.array_equal(g, want[f"arr_{i}"], equal_nan=True), i


def test_captured_gpt_forward_follows_the_weights():
    """The caller captures a forward (and a training step): whatever was current on the host at capture time, a replay must use
    the weights of the moment it runs, and an eager forward those that replays have left."""
    from deers_b200 import gpt
    from oracle import ref
    V, L, H, C, Hm, T, B = 1100, 1, 2, 64, 128, 24, 1                     # the head on the tensor core
    cfg = (V, L, H, C, Hm)
    rng = np.random.default_rng(21)
    ids, tgt = (torch.from_numpy(rng.integers(0, V, (B, T))).cuda() for _ in range(2))

    def model(seed):
        m = gpt.GPT(gpt.GPTConfig(V, T, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
        m.load_parameters(ref.gpt_init_params(cfg, seed=seed))
        return m

    def captured(m, fn):
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=m.stream):
            out = fn()
        return g, out

    def check(m, got, what):
        torch.cuda.synchronize()
        want = ref.gpt_step(cfg, [m.parameter(i) for i in range(m.num_parameters())], ids.cpu().numpy(), want_grads=False)["logits"]
        assert_close(got.cpu().numpy().reshape(np.asarray(want).shape), want, 1e-4, what)      # f32 sums of up to 128 terms

    # captured when the head's pair is current; replayed after a step, an upload, a step on the same model
    m = model(31)
    check(m, m.forward(ids), "eager")
    g, out = captured(m, lambda: m.forward(ids))
    g.replay()
    check(m, out, "replay")
    m.train_step(ids, tgt, lr=1e-1)
    g.replay()
    check(m, out, "replay after a step")
    check(m, m.forward(ids), "eager after a replay")
    m.load_parameters(ref.gpt_init_params(cfg, seed=32))
    g.replay()
    check(m, out, "replay after an upload")
    # captured when the pair has never been made; the first eager forward runs before any replay
    m = model(33)
    g, out = captured(m, lambda: m.forward(ids))
    check(m, m.forward(ids), "eager after a capture")
    g.replay()
    check(m, out, "first replay")
    # forward and backward captured, then an eager forward
    m = model(34)
    g, out = captured(m, lambda: m.forward_backward(ids, tgt))
    check(m, m.forward(ids), "eager after a captured backward")
    # a captured training step moves the weights without a call
    m = model(35)
    m.forward(ids)
    g, out = captured(m, lambda: m.train_step(ids, tgt, lr=1e-1))
    check(m, m.forward(ids), "eager before the replay")
    g.replay()
    check(m, m.forward(ids), "eager after a replayed step")
    g.replay()
    check(m, m.forward(ids), "eager after two replayed steps")


def test_gpt_forward_costs_what_its_tokens_cost():
    """A length seen for the first time goes the way of every other (the same launches in every call), and a batch of short
    sequences computes its tokens, not whole blocks of them."""
    from deers_b200 import gpt
    V, L, H, C, Hm, T, B = 8192, 2, 4, 128, 512, 64, 256
    m = gpt.GPT(gpt.GPTConfig(V, T, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    ids = torch.zeros((B, T), dtype=torch.int64, device="cuda")
    m.forward(ids)                                                          # makes the head's pair
    for t in (5, 6, 37):
        part, counts = ids[:3, :t].contiguous(), []
        for _ in range(4):
            before = m.ctx.launch_count()
            m.forward(part)
            counts.append(m.ctx.launch_count() - before)
        assert len(set(counts)) == 1, counts

    def ms(t):
        part, best = ids[:, :t].contiguous(), float("inf")
        for _ in range(6):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            m.forward(part)
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        return best
    assert ms(33) < 0.8 * ms(64)                                            # 0.52 of the tokens


@pytest.mark.parametrize("M,N,K", [(3_000_000, 32, 256), (4_300_000, 128, 8), (4_200_001, 3, 5)])
def test_f32_gemm_more_tile_rows_than_a_grid_has(M, N, K):
    """Row tiles beyond 65535, with the tile variants a narrow and a wider product take."""
    from deers_b200 import gpt
    gen = torch.Generator(device="cuda").manual_seed(K)
    a, b = torch.randn((M, K), device="cuda", generator=gen), torch.randn((K, N), device="cuda", generator=gen)
    got = gpt.gemm_f32(a, b)
    worst = 0.0
    for r in range(0, M, 1 << 19):
        want = a[r:r + (1 << 19)].double() @ b.double()
        worst = max(worst, (got[r:r + (1 << 19)].double() - want).abs().max().item())
    # K products of unit normals: partial sums stay within 6 sqrt(K), each of the K additions rounds by 2^-24 of that
    assert worst <= 6.0 * K ** 0.5 * K * 2.0 ** -24


def test_f32_attention_backward_of_the_longest_sequence():
    """T = 2^20 has as many row tiles as the grid can hold.  With K = 0 the weights of row i are 1 / (i + 1), with V = 1 the
    output is 1 and dS is 0, so every result has a closed form."""
    from deers_b200 import ops
    T, D = 1 << 20, 4
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, do = (torch.randn((1, 1, T, D), device="cuda", generator=gen) for _ in range(2))
    k, v = torch.zeros_like(q), torch.ones_like(q)
    n = torch.arange(1, T + 1, dtype=torch.float64, device="cuda")
    dq, dk, dv = ops.attention_bwd(q, k, v, torch.ones_like(q), n.log().float()[None, None], do, ops.default_scale(D))
    assert dq.abs().max() == 0.0
    want = torch.flip(torch.cumsum(torch.flip(do[0, 0].double() / n[:, None], (0,)), 0), (0,))
    # weights carry the rounding of lse * log2(e) (14 * 2^-23); a group adds 2^18 terms whose magnitudes sum to 3.5 ln(T) at
    # most, and the errors of the additions add up like a random walk
    assert (dv[0, 0].double() - want).abs().max() <= (14 * 2.0 ** -23 + 2.0 ** 9 * 2.0 ** -24) * 3.5 * 14
    # dS = P (dP - delta): two sums of D products that cancel up to their rounding, times Q
    assert dk.abs().max() <= 2 * D * 2.0 ** -24 * 6 * 14 * 6


def test_other_threads_run_while_a_launch_waits():
    """A launch blocks while the device's queue is full.  The operators hold no interpreter lock then: a second thread keeps
    ticking; and two threads that share a stream get the results of one."""
    import threading
    import time
    from deers_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn((1, 4, t, 64), device="cuda", generator=gen).half() for t in (1, 256, 256))
    want = ops.attention_decode(q, k, v)
    x, w = torch.randn((64, 64), device="cuda", generator=gen).half(), torch.randn((64, 64), device="cuda", generator=gen).half()
    want_y = ops.Linear.new(x, w).forward()
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), [0.0]

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(1e-3)
            now = time.perf_counter()
            gaps[0], last = max(gaps[0], now - last), now
    t = threading.Thread(target=tick)
    t.start()
    begin = time.perf_counter()
    torch.cuda._sleep(1_500_000_000)                                        # about 0.8 s of an idle kernel in front
    outs = [ops.attention_decode(q, k, v) for _ in range(3000)]             # more than the queue holds
    waited = time.perf_counter() - begin
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    assert waited > 0.4, "the queue never filled: nothing was tested"
    assert gaps[0] < 0.25 * waited, (gaps[0], waited)

    wrong = []

    def work():
        for _ in range(300):
            o, y = ops.attention_decode(q, k, v), ops.Linear.new(x, w).forward()
            if not (torch.equal(o, want) and torch.equal(y, want_y)):
                wrong.append(1)
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def backward_peak(call):
    """Bytes a call takes at its peak beyond what was held before it."""
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = call()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - before, out


def test_backward_weighs_its_workspace_against_the_memory_of_the_moment():
    """The larger workspace is taken when it is at most a quarter of what is free: after a call that took it on an empty device,
    one on a nearly full device must not; memory that torch's allocator holds unused counts as free."""
    from deers_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v, do = (torch.randn((2, 16, 8192, 64), device="cuda", generator=gen).half() for _ in range(4))
    scale = ops.default_scale(64)
    o, lse = ops.attention_fwd(q, k, v, scale)
    least, fast = (ops.workspace_bytes(q, scale, True, p) for p in (1, 2))
    grads = 3 * q.numel() * 2
    assert fast > torch.cuda.get_device_properties(0).total_memory // 512
    torch.cuda.empty_cache()
    peak, want = backward_peak(lambda: ops.attention_bwd(q, k, v, o, lse, do, scale))
    assert peak >= fast + grads                                             # empty device: kept dS
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - 2 * fast, dtype=torch.uint8, device="cuda")
    peak, got = backward_peak(lambda: ops.attention_bwd(q, k, v, o, lse, do, scale))
    assert peak < least + grads + (8 << 20), (peak, least, fast)            # half of what is left: recomputed
    for a, b in zip(got, want):                                             # f16 rounding of the same dS values
        assert_close(a.float().cpu().numpy(), b.float().cpu().numpy(), TOL_F16, "gradients")
    del fill                                                                # unused, and still the allocator's
    peak, got = backward_peak(lambda: ops.attention_bwd(q, k, v, o, lse, do, scale))
    assert peak >= fast + grads
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    del got, want
    torch.cuda.empty_cache()


@pytest.mark.parametrize("D,T", [(8, 129), (56, 300), (72, 127), (80, 385), (120, 257)])
@pytest.mark.parametrize("causal", [True, False])
def test_f16_recomputing_backward_at_other_head_dims(D, T, causal):
    """A workspace of the two statistics arrays and nothing else, which head dims between the tile widths may be given too:
    the kernel that recomputes S and dP must run, in that workspace, on several and on ragged tiles."""
    from deers_b200 import ops
    from oracle import ref
    B, H = 2, 3
    rng = np.random.default_rng(D * T)
    host = [rng.standard_normal((B, H, T, D)).astype(np.float16).astype(np.float32) for _ in range(4)]
    q, k, v, do = (torch.from_numpy(a).to("cuda", torch.float16) for a in host)
    scale = ops.default_scale(D)
    o, lse = ops.attention_fwd(q, k, v, scale, causal)
    bytes_used = ops.workspace_bytes(q.new_empty((B, H, T, 64 if D < 64 else 128)), scale, causal, 1)
    assert bytes_used == 2 * B * H * -(-T // 128) * 128 * 4 < ops.workspace_bytes(q, scale, causal, 1)
    ws = torch.full((bytes_used + 256,), 0xFF, dtype=torch.uint8, device="cuda")
    taken, got = backward_peak(lambda: ops.attention_bwd(q, k, v, o, lse, do, scale, causal, workspace=ws[:bytes_used]))
    assert taken <= 3 * (q.numel() * 2 + 512), "a workspace of its own beside the caller's"
    assert torch.all(ws[bytes_used:] == 0xFF)
    want = ref.attn_fwd_bwd(*host, causal=causal)
    for name, g, w in zip(("dq", "dk", "dv"), got, want[2:]):
        assert_close(g.float().cpu().numpy(), w, TOL_F16, f"D {D} T {T} {name}")


def test_backward_allocates_what_its_kernels_use():
    from deers_b200 import ops
    q, k, v, do = (torch.randn((4, 8, 1000, 80), device="cuda").half() for _ in range(4))
    o, lse = ops.attention_fwd(q, k, v, ops.default_scale(80))
    fast = ops.workspace_bytes(q.new_empty((4, 8, 1000, 128)), pass_=2)
    taken, _ = backward_peak(lambda: ops.attention_bwd(q, k, v, o, lse, do, ops.default_scale(80)))
    # three gradients and 36 dS tiles of 32 KB for each of 32 slices; the allocator rounds each up to 2 MB at most
    assert taken <= 3 * q.numel() * 2 + fast + 4 * (2 << 20), (taken, fast)


def test_a_failed_call_leaves_no_error_for_the_next():
    """A stream whose recording has been invalidated refuses every launch, on the host.  The call that meets it answers with the
    error; the next call, on a stream that is well, has none."""
    import ctypes

    from deers_b200 import _lib, ops
    rt, L = ctypes.CDLL("libcudart.so.12"), _lib.lib()                      # the runtime torch has loaded
    a, b, c = (torch.ones((64, 64), device="cuda") for _ in range(3))
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        sick = ops.Context.current(a.device)
    well = ops.Context.current(a.device)
    assert sick.handle != well.handle

    def product(ctx):
        return L.deers_b200_gemm_f32(ctx.handle, 64, 64, 64, a.data_ptr(), 64, 0, b.data_ptr(), 64, 1, c.data_ptr(), 64, None, None, 0)

    assert product(well) == _lib.OK and product(sick) == _lib.OK
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(ctypes.c_void_p(st.cuda_stream), 2) == 0
    assert rt.cudaStreamSynchronize(ctypes.c_void_p(st.cuda_stream)) != 0   # not allowed while recording: invalidates it
    assert product(sick) == _lib.ERR_CUDA
    assert product(well) == _lib.OK
    graph = ctypes.c_void_p()
    assert rt.cudaStreamEndCapture(ctypes.c_void_p(st.cuda_stream), ctypes.byref(graph)) != 0 and not graph.value
    rt.cudaGetLastError()
    assert product(sick) == _lib.OK and product(well) == _lib.OK
    torch.cuda.synchronize()
    assert torch.all(c == 64.0)


def test_f16_tensors_off_a_16_byte_boundary():
    """A view that starts anywhere is compacted; a contiguous tensor that does, or a head_dim there are no tiles for, is refused
    with the library's own status."""
    from deers_b200 import _lib, ops
    from deers_b200.errors import CudaError
    B, H, T, D = 1, 2, 20, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    good = torch.randn((B, H, T, D), dtype=torch.float16, device="cuda", generator=g)
    wide = torch.randn((B, H, T, D + 8), dtype=torch.float16, device="cuda", generator=g)
    view = wide[..., 1:D + 1]
    off = torch.randn(B * H * T * D + 1, dtype=torch.float16, device="cuda", generator=g)[1:].view(B, H, T, D)
    scale = ops.default_scale(D)
    o, lse = ops.attention_fwd(view, good, good, scale)
    o2, lse2 = ops.attention_fwd(view.contiguous(), good, good, scale)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
    for call in (lambda: ops.attention_fwd(off, good, good, scale), lambda: ops.attention_bwd(good, good, off, o, lse, good, scale)):
        with pytest.raises(CudaError) as e:
            call()
        assert e.value.status == _lib.ERR_LAYOUT
    x = torch.zeros((1, 2, 4, 100), dtype=torch.float16, device="cuda")
    for call in (lambda: ops.attention_fwd(x, x, x, scale), lambda: ops.attention_bwd(x, x, x, x, lse, x, scale)):
        with pytest.raises(CudaError) as e:
            call()
        assert e.value.status == _lib.ERR_SHAPE


@pytest.mark.parametrize("dtype,D,Tk,Tq", [(torch.float16, 80, 2, 1), (torch.float16, 64, 9, 1), (torch.float16, 128, 40, 3),
                                           (torch.float32, 56, 17, 17), (torch.float16, 96, 700, 1), (torch.float32, 128, 3000, 2)])
def test_decode_nan_and_inf_scores(dtype, D, Tk, Tq):
    """A NaN in a key is in the result of every query that sees it, also where the lanes that hold the key hold no other; a
    score of -inf is a weight of zero."""
    from deers_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(Tk)
    q = torch.rand((2, 2, Tq, D), device="cuda", generator=g).to(dtype) + 0.5
    k, v = (torch.randn((2, 2, Tk, D), device="cuda", generator=g).to(dtype) for _ in range(2))
    for j in sorted({0, 1, Tk // 2, Tk - 1}):
        sees = torch.arange(Tq, device="cuda") + Tk - Tq >= j
        bad = k.clone()
        bad[1, 0, j, D - 1] = float("nan")
        o, lse = ops.attention_decode(q, bad, v, want_lse=True)
        want = torch.zeros((2, 2, Tq), dtype=torch.bool, device="cuda")
        want[1, 0] = sees
        assert torch.equal(lse.isnan(), want) and torch.equal(o.isnan(), want[..., None].expand_as(o)), j
        bad[1, 0, j, D - 1] = float("-inf")
        o = ops.attention_decode(q, bad, v)
        alone = Tq == Tk and j == 0                                         # the first query sees nothing else: 0 / 0
        s = (q.double() @ k.double().transpose(2, 3)) / D ** 0.5
        s[1, 0, :, j] = float("-inf")
        s = s.masked_fill(torch.ones(Tq, Tk, dtype=torch.bool, device="cuda").triu(Tk - Tq + 1), float("-inf"))
        exact = s.softmax(-1) @ v.double()
        assert torch.equal(o.isnan(), exact.isnan()) and bool(exact.isnan().any()) == alone, j
        assert_close(o.nan_to_num().float().cpu().numpy(), exact.nan_to_num().cpu().numpy(), TOL_F16 if dtype == torch.float16 else 1e-4, f"{j}")


@pytest.mark.parametrize("B,H,T,D", [(1, 1, 128, 32), (1, 1, 129, 32), (4, 6, 256, 32), (10, 4, 255, 16), (3, 13, 241, 30), (1, 2, 300, 32),
                                     (1, 1, 513, 20), (1, 3, 257, 64), (2, 3, 200, 52)])
@pytest.mark.parametrize("causal", [True, False])
def test_f32_attention_group_counts(B, H, T, D, causal):
    """Four or eight groups per block, tiles of 32 or 64 keys: by sequence length, head width and number of blocks."""
    from deers_b200 import ops
    from oracle import ref
    from tests.helpers import TOL_F32
    rng = np.random.default_rng(T * 17 + D)
    host = [rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4)]
    q, k, v, do = (torch.from_numpy(a).cuda() for a in host)
    op = ops.CausalAttention.new(q, k, v, None, causal)
    o = op.forward()
    grads = ops.GradientStore()
    op.backward(grads, do)
    ops.Context.current(q.device).sync()
    want = ref.attn_fwd_bwd(*host, causal=causal)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), [o, op.lse] + [grads.get(t) for t in (q, k, v)], want):
        assert_close(g.cpu().numpy(), w, TOL_F32, f"B {B} H {H} T {T} D {D} {name}")


@pytest.mark.parametrize("V,L,H,D,Hm,B,T", [
    (1031, 2, 2, 48, 100, 2, 33),      # 96 wide tiles, the ones for such heads, cost too much here; odd vocabulary, dense logits off 16-byte boundaries
    (1024, 1, 3, 32, 64, 1, 129),      # heads that fit every tile
    (50, 2, 2, 12, 20, 2, 17),         # halves of six: no rotation inside the kernels, on either side
    (61, 1, 4, 24, 36, 3, 20), (1100, 2, 2, 80, 64, 2, 40),              # ... no tile holds heads of 80 whole; backward rotates
    (1033, 3, 5, 16, 60, 1, 70), (1040, 1, 2, 128, 513, 1, 65), (37, 0, 2, 8, 5, 1, 9)])
def test_gpt_norms_rotations_and_grouped_gradients(V, L, H, D, Hm, B, T):
    """Head widths, depths and sizes at which norm, rotation, logits and weight gradients take another route."""
    from deers_b200 import gpt
    from oracle import ref
    C = H * D
    cfg = (V, L, H, C, Hm)
    params = ref.gpt_init_params(cfg, seed=3)
    rng = np.random.default_rng(V + T)
    ids, tgt = rng.integers(0, V, (B, T)), rng.integers(0, V, B * T)
    m = gpt.GPT(gpt.GPTConfig(V, T, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    m.load_parameters(params)
    tid, ttg = torch.from_numpy(ids).cuda(), torch.from_numpy(tgt).cuda()
    logits = m.forward(tid)
    loss = m.forward_backward(tid, ttg)
    again = m.forward(tid)
    m.ctx.sync()
    want = ref.gpt_step(cfg, params, ids, tgt)
    got = logits.cpu().numpy().reshape(B * T, V)
    assert np.isfinite(got).all() and torch.equal(logits, again)
    assert np.abs(got - want["logits"]).max() <= 1e-4 * np.abs(want["logits"]).max()
    assert abs(loss.item() - want["loss"]) < 1e-5 * max(1.0, abs(want["loss"]))
    for i in range(2 + 6 * L):
        g, w = m.grad(i), want["grads"][i]
        assert np.abs(g - w).max() <= 1e-4 * np.abs(w).max() + 1e-7, m.parameter_info(i)


def _gpt_and_oracle(V, L, H, D, Hm, B, T):
    """A model with its gradients made and the oracle's step on the same batch: (model, ids, targets, logits, loss, launches of the
    forward and of forward_backward, the oracle's results)."""
    from deers_b200 import gpt
    from oracle import ref
    cfg = (V, L, H, H * D, Hm)
    params = ref.gpt_init_params(cfg, seed=5)
    rng = np.random.default_rng(V + T)
    ids, tgt = rng.integers(0, V, (B, T)), rng.integers(0, V, B * T)
    m = gpt.GPT(gpt.GPTConfig(V, T, L, H, H * D, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    m.load_parameters(params)
    tid, ttg = torch.from_numpy(ids).cuda(), torch.from_numpy(tgt).cuda()
    m.forward(tid)
    at = [m.ctx.launch_count()]
    logits = m.forward(tid)
    at.append(m.ctx.launch_count())
    loss = m.forward_backward(tid, ttg)
    at.append(m.ctx.launch_count())
    m.ctx.sync()
    return m, tid, ttg, logits, loss, (at[1] - at[0], at[2] - at[1]), ref.gpt_step(cfg, params, ids, tgt)


def _check_gpt(m, logits, loss, want):
    """f32 sums on either side: 1e-4 of the largest value, as for the other models."""
    got = logits.cpu().numpy().reshape(want["logits"].shape)
    assert np.abs(got - want["logits"]).max() <= 1e-4 * np.abs(want["logits"]).max()
    assert abs(loss.item() - want["loss"]) < 1e-5 * max(1.0, abs(want["loss"]))
    for i, w in enumerate(want["grads"]):
        assert np.abs(m.grad(i) - w).max() <= 1e-4 * np.abs(w).max() + 1e-7, m.parameter_info(i)


@pytest.mark.parametrize("H,D,Hm,B,T,launches", [(4, 32, 512, 2, 40, 1), (6, 32, 768, 1, 70, 1), (5, 64, 1280, 2, 35, 4), (4, 128, 300, 1, 33, 4)])
def test_gpt_weight_gradients_in_one_launch_or_apart(H, D, Hm, B, T, launches):
    """One launch per block where that is one wave of blocks, four where it would be several; the second stream changes no bit."""
    fwd, step = [], []
    for L in (1, 3):
        m, ids, tgt, logits, loss, n, want = _gpt_and_oracle(64, L, H, D, Hm, B, T)
        fwd.append(n[0]), step.append(n[1])
        _check_gpt(m, logits, loss, want)
    # of a block's backward: three input gradients, two norms, the attention, the input gradient of the projection
    assert (step[1] - step[0]) - (fwd[1] - fwd[0]) == 2 * (7 + launches)
    grads = [m.grad(i) for i in range(m.num_parameters())]
    m.ctx.kernel_timing(True)                                     # everything on one stream
    m.forward_backward(ids, tgt)
    m.ctx.sync()
    m.ctx.kernel_timing(False)
    for i, g in enumerate(grads):
        assert np.array_equal(g, m.grad(i)), m.parameter_info(i)


@pytest.mark.parametrize("H,D,B,T,tile", [
    # the projection's tile and whether blocks of a cluster share its K
    (6, 32, 1, 100, (16, 32, 0)), (20, 16, 1, 64, (16, 32, 0)), (21, 16, 1, 2, (16, 32, 1)),
    (1, 16, 5, 239, (32, 32, 0)), (15, 32, 1, 19, (32, 32, 1)),
    (2, 64, 1, 4, (32, 64, 0)), (16, 16, 3, 100, (32, 64, 0)), (4, 64, 1, 4, (32, 64, 1)), (6, 64, 1, 3, (32, 64, 1)),
    (2, 64, 4, 250, (64, 64, 0)), (5, 64, 2, 66, (64, 64, 1)),
    (1, 48, 1, 4, (32, 96, 0)), (5, 48, 1, 196, (32, 96, 1)),
    (5, 24, 5, 239, (64, 96, 0)), (13, 48, 1, 33, (64, 96, 1)),
    (4, 128, 1, 584, (64, 128, 0)), (17, 32, 1, 175, (64, 128, 1)),
    (12, 32, 1, 700, (128, 64, 0)), (5, 64, 1, 932, (128, 64, 0)),            # the tensor core's
    (20, 16, 3, 100, (128, 64, 1)), (5, 32, 2, 320, (128, 64, 1)), (6, 64, 1, 281, (128, 64, 1)),
    # no tile holds the heads, or such tiles cost more than a launch, or they would be several waves of clusters
    (3, 80, 1, 40, None), (3, 10, 2, 25, None), (4, 48, 1, 231, None), (2, 96, 1, 100, None), (8, 64, 1, 256, None)])
def test_gpt_rotation_inside_the_projection(H, D, B, T, tile):
    """Norm and rotation in each tile of the projection, whole K and K split over a cluster (the other half of a head and the rows'
    squares then lie in several blocks)."""
    inside = tile is not None
    r = _route(_lib.PRODUCT_F32_NORM, B * T, 3 * H * D, H * D, aligned=H * D % 4 == 0, heads=D)
    assert r.rotated == inside and (not inside or (r.tile_m, r.tile_n, r.parts > 1) == tile)
    m, ids, tgt, logits, loss, n, want = _gpt_and_oracle(64, 1, H, D, 64, B, T)
    _check_gpt(m, logits, loss, want)
    # embedding; projection, attention, output, up, down (and the rotation); norm, head, copy of its padded rows
    assert n[0] == 1 + 5 + (not inside) + 3


@pytest.mark.parametrize("H,D,Hm,B,T,parts", [(7, 64, 2048, 1, 130, 2), (8, 64, 2048, 1, 260, 1), (10, 64, 1024, 2, 258, 1), (40, 10, 1500, 1, 260, 2)])
def test_gpt_up_projection_of_wide_models_on_the_tensor_core(H, D, Hm, B, T, parts):
    """Norm and product of an up projection, which rotates nothing, whatever its width; whole K and K shared by a cluster.  (Heads of ten columns: the
    other norm's product rotates nothing either.)"""
    C = H * D
    r = _route(_lib.PRODUCT_F32_NORM, B * T, Hm, C)
    assert (r.tensor_core, r.parts, r.rotated) == (1, parts, 0)
    if D % 8:
        assert _route(_lib.PRODUCT_F32_NORM, B * T, 3 * C, C, heads=D).tensor_core
    m, ids, tgt, logits, loss, n, want = _gpt_and_oracle(64, 1, H, D, Hm, B, T)
    _check_gpt(m, logits, loss, want)


def test_gpt_train_step_takes_pointers_on_any_boundary():
    """What a copy takes and a kernel cannot: ids four bytes off their boundary, loss and norm one byte off."""
    import ctypes
    from deers_b200 import _lib, gpt
    from oracle import ref
    V, T, B = 40, 9, 2
    cfg = (V, 1, 2, 16, 24)
    params = ref.gpt_init_params(cfg, seed=1)
    rng = np.random.default_rng(2)
    ids, tgt = (torch.from_numpy(rng.integers(0, V, B * T)).cuda() for _ in range(2))
    said = []
    for off, out_off in ((0, 0), (4, 1)):
        m = gpt.GPT(gpt.GPTConfig(V, T, 1, 2, 16, 24), ids.device, B)
        m.load_parameters(params)
        buf = torch.zeros(2 * (8 * B * T + 8) + 24, dtype=torch.uint8, device="cuda")
        ia, ta, oa = off, 8 * B * T + 8 + off, 2 * (8 * B * T + 8) + out_off
        buf[ia:ia + 8 * B * T] = ids.view(torch.uint8)
        buf[ta:ta + 8 * B * T] = tgt.view(torch.uint8)
        torch.cuda.synchronize()
        h = _lib.AdamWHyper(1e-3, 0.9, 0.999, 1e-8, 0.1, 1)
        p = buf.data_ptr()
        assert _lib.lib().deers_b200_gpt_train_step(m.handle, p + ia, p + ta, B, T, ctypes.byref(h), 1.0, p + oa, p + oa + 4) == _lib.OK
        m.ctx.sync()
        said.append((buf[oa:oa + 8].cpu().numpy().tobytes(), [m.parameter(i) for i in range(m.num_parameters())]))
    assert said[0][0] == said[1][0] and np.isfinite(np.frombuffer(said[0][0], np.float32)).all()
    assert all(np.array_equal(a, b) for a, b in zip(said[0][1], said[1][1]))


@pytest.mark.parametrize("V,L,H,D,Hm,B,T", [
    (1024, 1, 12, 86, 64, 1, 5),       # rows of 1032: a block each, in the backward with the normalised row and in the head's f16 pair
    (1031, 0, 82, 100, 8, 2, 3),       # rows of 8200: no pair in one pass, the head normalises and splits
    (40, 1, 82, 100, 16, 1, 3),        # ... and two passes of 16-byte loads in the backward
    (1024, 2, 3, 10, 21, 2, 9)])       # rows of 30: element by element everywhere
def test_gpt_norms_of_wide_and_ragged_rows(V, L, H, D, Hm, B, T):
    m, ids, tgt, logits, loss, n, want = _gpt_and_oracle(V, L, H, D, Hm, B, T)
    _check_gpt(m, logits, loss, want)


@pytest.mark.parametrize("n,V,C", [(1, 1, 5), (257, 2, 24), (1023, 40, 33), (1025, 3, 8), (2600, 7, 2049), (3000, 100000, 16)])
def test_embedding_backward_of_repeated_ids(n, V, C):
    """Ids that repeat within and across the 1024 looked at together, up to every token the same: the sum in token order, bit for bit."""
    from deers_b200 import gpt
    from oracle import ref
    rng = np.random.default_rng(n)
    ids, d = rng.integers(0, V, n), rng.standard_normal((n, C)).astype(np.float32)
    got = gpt.embedding_backward(torch.from_numpy(d).cuda(), torch.from_numpy(ids).cuda(), V)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy(), ref.embedding_bwd(d, ids, V))


def _route(which, M, N, K, a_mn=False, b_mn=True, aligned=True, heads=0):
    """How a product would run: a test of one route asks, or a change of the choice would leave it testing another."""
    from deers_b200 import ops
    return ops.Context.current(torch.device("cuda", torch.cuda.current_device())).product_route(which, [(M, N)], K, a_mn, b_mn, aligned, heads)


@pytest.mark.parametrize("M,N,K,pair", [(*size, False) for size in (
    (256, 256, 64), (264, 264, 328), (520, 192, 1032), (512, 520, 8192), (640, 1544, 4104), (1280, 768, 8192), (2056, 2304, 776), (4104, 1288, 200), (8192, 96, 72),
    (9472, 768, 64), (304, 3000, 16392), (4104, 2056, 72), (2184, 4488, 1032))] + [(*size, True) for size in (
    (9480, 4864, 264), (8072, 2264, 776), (7992, 2104, 1032), (3848, 4472, 776), (4744, 3832, 840))])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_f16_gemm_pairs_of_ctas(M, N, K, pair, a_mn, b_mn):
    """Tiles of 256 rows by two CTAs: a second half of few or no rows, columns that end in either half, fewer K blocks than stages and more, several tiles a
    pair; and sizes near them that stay with single CTAs.  Small integers, as above; sums of up to 16392 terms of which few are not zero."""
    assert _route(_lib.PRODUCT_F16, M, N, K, a_mn, b_mn).pair == pair
    from deers_b200 import ops
    rng = np.random.default_rng(M + N + K)
    a = rng.integers(-1, 2, (K, M) if a_mn else (M, K)).astype(np.float16)
    b = rng.integers(-1, 2, (K, N) if b_mn else (N, K)).astype(np.float16)
    a *= rng.random(a.shape) < 0.3
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    got = ops._gemm(M, N, K, ta, int(a_mn), tb, int(b_mn))
    ops.Context.current(got.device).sync()
    want = (ta.float().T if a_mn else ta.float()).double() @ (tb if b_mn else tb.T).double()
    assert want.abs().max().item() <= 2048
    assert torch.equal(got.double(), want)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (False, False), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K,tensor_core", [
    (2052, 1540, 4, "aligned"), (1156, 1028, 20, "no"), (2048, 640, 64, "no"), (1028, 1092, 68, "aligned"), (1100, 644, 132, "yes"), (1024, 768, 192, "yes"),
    (1284, 196, 1000, "yes"), (260, 1540, 772, "yes"), (196, 772, 2052, "yes"),
    (1660, 508, 4, "yes"), (1404, 636, 20, "yes"), (1276, 700, 64, "yes"), (636, 956, 68, "yes")])
def test_f32_gemm_on_the_tensor_core(M, N, K, tensor_core, a_mn, b_mn, aligned):
    """Tiles that end in rows, columns and k, one short stage to many, whole K and K shared by a cluster, each storage order, rows on 16-byte
    boundaries and on none.  Values of three bf16 each, sums that start anew every 16 k: 1e-7 of the result in the 2-norm (measured 5e-8 to
    8.1e-8; two f16 per value or one accumulator give 2.8e-7), and small integers exactly."""
    from deers_b200 import gpt
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    pad = 0 if aligned else 1

    def operand(rows, cols, whole):
        t = torch.empty((rows, cols + pad), device="cuda")
        t.copy_(torch.randint(-8, 9, t.shape, device="cuda", generator=g) if whole else torch.randn(t.shape, device="cuda", generator=g))
        return t[:, pad:]

    assert _route(_lib.PRODUCT_F32, M, N, K, a_mn, b_mn, aligned).tensor_core == (tensor_core == "yes" or tensor_core == "aligned" and aligned)
    for whole in (False, True):
        a = operand(*((K, M) if a_mn else (M, K)), whole)
        b = operand(*((K, N) if b_mn else (N, K)), whole)
        got = gpt.gemm_f32(a, b, a_mn, b_mn)
        again = gpt.gemm_f32(a, b, a_mn, b_mn)
        want = (a.double().T if a_mn else a.double()) @ (b.double() if b_mn else b.double().T)
        assert torch.equal(got, again)
        if whole:
            assert torch.equal(got.double(), want)
        else:
            assert ((got.double() - want).norm() / want.norm()).item() < 1e-7


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("small", ["a", "b"])
@pytest.mark.parametrize("power", [-99, -112])
def test_f32_gemm_on_the_tensor_core_of_small_values(power, small, aligned):
    """One operand times 2^-99 or 2^-112, the other times 2^64, no value of the unscaled ones below 2^-12.  The three parts hold every bit of a value;
    from 2^-111 on its two leading parts are full, and all are the unscaled ones times a power of two: bit for bit the unscaled result so scaled.  Smaller
    values have fewer bits in the leading parts and more in the last: 1e-7 in the 2-norm as for other operands (measured 5.8e-8 scaled and not)."""
    from deers_b200 import gpt
    M, N, K = 1024, 768, 192
    g = torch.Generator(device="cuda").manual_seed(9)
    a, b = (torch.randn((r, c + (not aligned)), device="cuda", generator=g)[:, int(not aligned):] for r, c in ((M, K), (K, N)))
    for t in (a, b):
        t[t.abs() < 2.0 ** -12] = 0.0
    base, want = gpt.gemm_f32(a, b, False, True).double(), a.double() @ b.double()
    a.mul_(2.0 ** (power if small == "a" else 64))
    b.mul_(2.0 ** (power if small == "b" else 64))
    got = gpt.gemm_f32(a, b, False, True).double() * 2.0 ** (-64 - power)
    assert ((got - want).norm() / want.norm()).item() < 1e-7
    if power == -99:
        assert torch.equal(got, base)


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,aligned", [(1024, 768, 192, 0, 1, 1), (1000, 768, 190, 1, 0, 0), (1024, 192, 768, 0, 0, 1)])
@pytest.mark.parametrize("small", ["a", "b"])
@pytest.mark.parametrize("power,other", [(-127, 100), (-130, 20), (-134, 100), (-138, 118), (-142, 24), (-146, 60)])
def test_f32_gemm_on_the_tensor_core_of_subnormal_operands(power, other, small, M, N, K, a_mn, b_mn, aligned):
    """An operand of subnormal values, the other one small or large, whole (as the second half of the rows or columns beside normal ones in the same
    tiles), K shared by a cluster, rows on any boundary.  Products of the two halves stand each for itself: a sum in f32 of at most K / 4 + 4 rounded
    terms of one size has a 2-norm error of about 2^-24 sqrt(K / 4) / 2, 2.1e-7 at K = 192 and 4.2e-7 at K = 768 (FFMA kernels measured 1.3e-7 at
    K = 192); the tensor core's six products alone gave 4.0e-6 at 2^-134 and 1.7e-3 at 2^-146."""
    from deers_b200 import gpt
    g = torch.Generator(device="cuda").manual_seed(power * power)
    a, b = (torch.randn(s, device="cuda", generator=g) for s in ((M, K), (K, N)))
    x, y = (a, b.T) if small == "a" else (b.T, a)
    x[x.shape[0] // 2:] *= 2.0 ** power
    y *= 2.0 ** other
    pad = 0 if aligned else 1
    store = [t.T if mn else t for t, mn in ((a, a_mn), (b.T, b_mn))]
    held = [torch.empty((t.shape[0], t.shape[1] + pad), device="cuda")[:, pad:].copy_(t) for t in store]
    got = gpt.gemm_f32(*held, bool(a_mn), bool(b_mn)).double()
    want = a.double() @ b.double()
    if small == "b":
        got, want = got.T, want.T
    half = x.shape[0] // 2
    assert _route(_lib.PRODUCT_F32, M, N, K, a_mn, b_mn, aligned).tensor_core
    assert ((got[:half] - want[:half]).norm() / want[:half].norm()).item() < 1e-7 * max(1.0, (K / 192) ** 0.5)
    assert ((got[half:] - want[half:]).norm() / want[half:].norm()).item() < 2.0 ** -25 * (K / 4) ** 0.5


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("M,N,K,a_mn,b_mn,aligned,parts", [(1024, 768, 192, False, True, True, 1), (1024, 768, 192, True, True, True, 1), (1024, 768, 192, False, False, True, 1),
                                                           (1024, 192, 768, False, True, True, 4), (1000, 770, 190, True, False, False, 1), (1001, 190, 770, False, True, False, 5)])
def test_f32_gemm_on_the_tensor_core_of_what_is_not_finite(value, M, N, K, a_mn, b_mn, aligned, parts):
    """Infinities, NaN and values that round to an infinity of bf16, in either operand and against zeros: what the products of f32 give.  One block a
    tile, and a cluster in which one block alone has them; rows on any boundary."""
    from deers_b200 import gpt
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = (torch.randn(s, device="cuda", generator=g) * 0.25 for s in ((M, K), (K, N)))
    a[700, 100], b[30, 5], b[100, 77] = value, value, 0.0
    r = _route(_lib.PRODUCT_F32, M, N, K, a_mn, b_mn, aligned)
    assert (r.tensor_core, r.parts) == (1, parts)
    pad = 0 if aligned else 1
    held = [torch.empty((t.shape[0], t.shape[1] + pad), device="cuda")[:, pad:].copy_(t) for t in (a.T if a_mn else a, b if b_mn else b.T)]
    got = gpt.gemm_f32(*held, a_mn, b_mn).double()
    want = a.double() @ b.double()
    assert torch.equal(got.isnan(), want.isnan())
    fin = want.abs() < 3e38
    assert torch.equal(got[~fin & ~want.isnan()].sign(), want[~fin & ~want.isnan()].sign())
    big = want[fin].abs() > 1e30
    assert (got[fin][~big] - want[fin][~big]).abs().max().item() < 1e-5
    assert ((got[fin][big] - want[fin][big]) / want[fin][big]).abs().nan_to_num(0).max().item() < 1e-5 if big.any() else True


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,tile,resident", [
    # logits: few waves, single CTAs
    (1024, 5008, 192, 0, 1, None, 0), (300, 12296, 64, 0, 1, None, 0), (2056, 2568, 256, 0, 1, None, 0), (520, 9608, 328, 0, 1, None, 0), (136, 20008, 24, 0, 1, None, 0),
    # many waves, pairs: A resident (one to four K blocks), and not (rows of tiles that would leave pairs idle, deeper K); rows that end in either half
    (1024, 12296, 64, 0, 1, (256, 128), 1), (1000, 12296, 128, 0, 1, (256, 128), 2), (136, 95000, 24, 0, 1, (256, 128), 1), (760, 18056, 192, 0, 1, (256, 128), 3),
    (2056, 6024, 256, 0, 1, (256, 128), 4), (1160, 9992, 64, 0, 1, (256, 128), 0), (1000, 12040, 328, 0, 1, (256, 128), 0),
    # input gradient: K shared out, 128 and 192 columns, one and two of them
    (1024, 192, 50264, 0, 0, (256, 192), 0), (264, 128, 30008, 0, 0, None, 0), (2000, 320, 16392, 0, 0, (256, 192), 0), (200, 64, 70000, 0, 0, (256, 128), 0),
    (520, 128, 40000, 0, 0, (256, 128), 0),
    # weight gradient, transposed: columns of the tile that are there in part, one to three of them; and few tokens or tiles, single CTAs
    (192, 50264, 1024, 1, 1, (192, 256), 0), (320, 50264, 520, 1, 1, (192, 256), 0), (576, 30008, 584, 1, 1, (192, 256), 0),
    (64, 40008, 264, 1, 1, None, 0), (320, 12296, 520, 1, 1, None, 0), (384, 30008, 72, 1, 1, None, 0)])
def test_f16x3_gemm_pairs_of_ctas(M, N, K, a_mn, b_mn, tile, resident):
    """The head's products by pairs of CTAs, and those near them that stay with single CTAs (tile None).  Operands of 22 bits (two f16), f32 sums in the
    tensor core: 2e-6 of the largest value times max(1, sqrt(K) / 16), as for single CTAs; small integers exactly, so any tile, half or K range
    dropped or taken twice shows."""
    r = _route(_lib.PRODUCT_F16X3, M, N, K, a_mn, b_mn)
    assert (r.pair, r.resident) == (tile is not None, resident) and (r.tile_m, r.tile_n) == (tile or (128, 128))
    from deers_b200 import gpt
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    for whole in (True, False):
        def operand(*shape):
            if whole:
                return torch.randint(-1, 2, shape, device="cuda", generator=g).float()
            return torch.randn(shape, device="cuda", generator=g)
        a, b = operand(*((K, M) if a_mn else (M, K))), operand(*((K, N) if b_mn else (N, K)))
        got = gpt.gemm_f16x3(a, b, bool(a_mn), bool(b_mn))
        again = gpt.gemm_f16x3(a, b, bool(a_mn), bool(b_mn))
        torch.cuda.synchronize()
        want = (a.double().T if a_mn else a.double()) @ (b.double() if b_mn else b.double().T)
        assert torch.equal(got, again)
        if whole:
            assert torch.equal(got.double(), want)
        else:
            assert (got.double() - want).abs().max().item() <= 2e-6 * max(1.0, K ** 0.5 / 16) * want.abs().max().item()


@pytest.mark.parametrize("V,H,D,B,T,pair,resident", [
    # a pass over the logits
    (12289, 2, 32, 2, 100, 0, 0), (50257, 6, 32, 1, 257, 0, 0), (9601, 5, 64, 3, 99, 0, 0), (10111, 4, 64, 2, 131, 0, 0), (1024, 2, 32, 1, 9, 0, 0),
    # statistics of the head product: one to four resident K blocks of A, deeper K, rows of tiles that would leave pairs idle; V that ends in a tile
    (131073, 1, 64, 1, 130, 1, 1), (50257, 2, 32, 2, 128, 1, 1), (24101, 4, 32, 2, 250, 1, 2), (12289, 6, 32, 4, 250, 1, 3), (12301, 4, 64, 4, 253, 1, 4),
    (24077, 5, 64, 2, 254, 1, 0), (9601, 6, 32, 5, 250, 1, 0)])
def test_gpt_cross_entropy_from_the_head_product(V, H, D, B, T, pair, resident):
    """Row statistics left by the head product or taken by a pass of their own: loss, logits (of an odd vocabulary: rows on any boundary, turned round in
    shared memory) and gradients of a model that is only embedding, norm and head, against float64.  The bound is the head products' (2e-6 of the
    largest value) with room for sums of V terms."""
    r = _route(_lib.PRODUCT_F16X3, B * T, V, H * D)
    assert (r.pair, r.resident) == (pair, resident)
    from deers_b200 import gpt
    C = H * D
    m = gpt.GPT(gpt.GPTConfig(V, T, 0, H, C, 8), torch.device("cuda", torch.cuda.current_device()), B)
    g = torch.Generator().manual_seed(V)
    wte, head = torch.randn((V, C), generator=g), torch.randn((C, V), generator=g) * 0.5
    m.load_parameters([wte.numpy(), head.numpy()])
    ids, tgt = torch.randint(0, V, (B, T), generator=g), torch.randint(0, V, (B, T), generator=g)
    tgt[0, 0], tgt[-1, -1] = 0, V - 1
    loss = m.forward_backward(ids.cuda(), tgt.cuda())
    m.ctx.sync()
    logits = m.forward(ids.cuda())
    w, h = wte.double().cuda().requires_grad_(), head.double().cuda().requires_grad_()
    x = w[ids.reshape(-1).cuda()]
    x = x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-5)
    exact = x @ h
    want = torch.nn.functional.cross_entropy(exact, tgt.reshape(-1).cuda())
    want.backward()
    assert abs(loss.item() - want.item()) < 1e-6 * max(1.0, want.item())
    assert (logits.reshape(-1, V).double() - exact).abs().max().item() <= 2e-6 * exact.abs().max().item()
    for i, t in enumerate((w, h)):
        assert np.abs(m.grad(i) - t.grad.cpu().numpy()).max() <= 1e-5 * t.grad.abs().max().item()


@pytest.mark.parametrize("scale,peak", [(1e-3, 0.0), (0.5, 0.0), (3.0, 0.0), (40.0, 0.0), (0.1, 20.0), (1.0, -30.0)])
def test_row_statistics_of_the_head_product(scale, peak):
    """Every token the same and every target the same, so that the mean loss is one row's: lse from the exponentials the head product's epilogue sums, for flat
    rows, rows of one large or one small logit and rows whose logits spread over hundreds (most exponentials zero), against float64 on the
    model's own logits.  log(s) + m, the picked logit less it and the mean round once each: 3 2^-24 of the largest of them.  s: an exponential is
    within 4 2^-24 of its value (two roundings of its argument's parts and the power of two), 32 of a thread are added in pairs and 3 more
    sums follow to 393 parts of 128 columns: 24 roundings of 2^-24."""
    from deers_b200 import gpt
    V, C, B, T = 50264, 64, 2, 128
    assert _route(_lib.PRODUCT_F16X3, B * T, V, C).pair
    m = gpt.GPT(gpt.GPTConfig(V, T, 0, 2, C, 8), torch.device("cuda", torch.cuda.current_device()), B)
    g = torch.Generator().manual_seed(7)
    wte, head = torch.randn((V, C), generator=g), torch.randn((C, V), generator=g) * scale
    for token in (0, 1, 77, V - 1):
        x = wte[token] / wte[token].square().mean().sqrt()
        head[:, 31 * token % V] = x * (peak / C) if peak else head[:, 31 * token % V]
    m.load_parameters([wte.numpy(), head.numpy()])
    for token in (0, 1, 77, V - 1):
        ids = torch.full((B, T), token, device="cuda")
        row = m.forward(ids)[0, 0].double()
        for t in (0, 31 * token % V, V - 1):
            loss = m.forward_backward(ids, torch.full((B, T), t, device="cuda")).item()
            want = (row.logsumexp(0) - row[t]).item()
            most = max(row.abs().max().item(), abs(want))
            assert abs(loss - want) <= 2.0 ** -24 * (3 * most + 28), (token, t)


def test_row_statistics_keep_a_nan_to_its_row():
    """One token's row of the embedding holds a NaN: its logits, its gradient and the mean loss are NaN, every other token's gradient is as it was."""
    from deers_b200 import gpt
    V, C, B, T = 50257, 64, 2, 128
    assert _route(_lib.PRODUCT_F16X3, B * T, V, C).pair
    m = gpt.GPT(gpt.GPTConfig(V, T, 0, 2, C, 8), torch.device("cuda", torch.cuda.current_device()), B)
    g = torch.Generator().manual_seed(3)
    wte, head = torch.randn((V, C), generator=g), torch.randn((C, V), generator=g) * 0.5
    ids = torch.randperm(V, generator=g)[:B * T].reshape(B, T)
    tgt = torch.randint(0, V, (B, T), generator=g).cuda()
    m.load_parameters([wte.numpy(), head.numpy()])
    m.forward_backward(ids.cuda(), tgt)
    m.ctx.sync()
    before = m.grad(0)[ids.reshape(-1).numpy()]
    wte[ids[1, 5], 9] = float("nan")
    m.load_parameters([wte.numpy(), head.numpy()])
    assert np.isnan(m.forward_backward(ids.cuda(), tgt).item())
    m.ctx.sync()
    after = m.grad(0)[ids.reshape(-1).numpy()]
    hit = T + 5
    assert np.isnan(after[hit]).all() and np.array_equal(np.delete(after, hit, 0), np.delete(before, hit, 0))


def test_gpt_products_of_values_that_are_infinite_in_bf16():
    """A channel of one head's values reaches 3.396e38 at the first token, which f32 holds and bf16 does not: the projection (with its norm), and the weight
    gradients in one launch, work out again what the tensor core's parts cannot hold.  Everything is finite; the gradients of the rows
    and columns concerned are compared each by its own size, as the other parameters are."""
    from deers_b200 import gpt, ops
    from oracle import ref
    V, L, H, D, Hm, B, T = 64, 1, 6, 32, 768, 4, 256
    C = H * D
    cfg = (V, L, H, C, Hm)
    params = [p.copy() for p in ref.gpt_init_params(cfg, seed=5)]
    m = gpt.GPT(gpt.GPTConfig(V, T, L, H, C, Hm), torch.device("cuda", torch.cuda.current_device()), B)
    at = {n: i for i, (n, _) in enumerate(m.named_parameters())}
    wte, wv, wo = (params[next(i for n, i in at.items() if k in n)] for k in ("wte", "v_proj", "out_proj"))
    channel, held = 5, 7
    wte[0, channel], wte[1:, channel] = 2.0, 0.0                 # (f32 attention sums before it divides: one such value, no overflow)
    n1 = wte[0] / np.sqrt((wte[0].astype(np.float64) ** 2).mean() + 1e-5)
    wv[:, held] = 0.0
    wv[channel, held] = np.float32(3.396e38 / n1[channel])
    wo[held] = np.random.default_rng(1).standard_normal(C).astype(np.float32) * np.float32(1e-37)
    rng = np.random.default_rng(2)
    ids, tgt = rng.integers(1, V, (B, T)), rng.integers(0, V, B * T)
    ids[:, 0] = 0
    m.load_parameters(params)
    route = m.ctx.product_route
    assert route(_lib.PRODUCT_F32_NORM, [(B * T, 3 * C)], C, heads=D).tensor_core
    assert route(_lib.PRODUCT_F32, [(Hm, C), (C, Hm), (C, C), (C, 3 * C)], B * T, True, True).tensor_core
    tid, ttg = torch.from_numpy(ids).cuda(), torch.from_numpy(tgt).cuda()
    logits, loss = m.forward(tid), m.forward_backward(tid, ttg)
    m.ctx.sync()
    want = ref.gpt_step(cfg, params, ids, tgt)
    got = logits.cpu().numpy().reshape(B * T, V)
    assert np.isfinite(want["logits"]).all() and np.abs(got - want["logits"]).max() <= 1e-4 * np.abs(want["logits"]).max()
    assert abs(loss.item() - want["loss"]) < 1e-5 * max(1.0, abs(want["loss"]))
    for name, i in at.items():
        g, w = m.grad(i), want["grads"][i]
        assert np.isfinite(w).all(), name
        if "out_proj" in name:
            assert np.abs(w[held]).max() > 1e30 and np.abs(g[held] - w[held]).max() <= 1e-4 * np.abs(w[held]).max()
            g, w = np.delete(g, held, 0), np.delete(w, held, 0)
        if "v_proj" in name:
            assert 0 < np.abs(w[:, held]).max() < 1e-35 and np.abs(g[:, held] - w[:, held]).max() <= 1e-4 * np.abs(w[:, held]).max()
            g, w = np.delete(g, held, 1), np.delete(w, held, 1)
        assert np.abs(g - w).max() <= 1e-4 * np.abs(w).max() + 1e-7, name


@pytest.mark.parametrize("B,H,T,D", [
    (1, 1, 2, 32), (1, 2, 7, 30), (1, 1, 8, 64), (2, 2, 9, 16), (1, 3, 33, 48), (1, 1, 257, 32), (1, 2, 200, 64), (1, 1, 90, 96), (1, 1, 70, 128),     # 8 rows a block
    (2, 5, 97, 32), (3, 4, 77, 48), (1, 6, 256, 32), (2, 8, 300, 30), (10, 4, 260, 16), (16, 4, 161, 32), (1, 12, 333, 20), (1, 2, 1000, 32), (1, 7, 130, 64), (1, 3, 300, 96), (2, 4, 100, 126)])         # 16 rows
@pytest.mark.parametrize("causal", [True, False])
def test_f32_attention_in_blocks_of_few_rows(B, H, T, D, causal):
    """Calls of few blocks, in blocks of 8 and 16 stationary rows: sequences that end inside a block and a streamed tile, both group counts, either
    direction (whose blocks may differ in size), widths off 16-byte boundaries.  (Not one key alone: its score gradient is the difference of
    two equal sums of D products, zero with a rounding of 2^-24 sqrt(D) times the largest product, and no value to hold that against.)"""
    from deers_b200 import ops
    from oracle import ref
    from tests.helpers import TOL_F32
    rng = np.random.default_rng(T * 19 + D)
    host = [rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4)]
    q, k, v, do = (torch.from_numpy(a).cuda() for a in host)
    op = ops.CausalAttention.new(q, k, v, None, causal)
    o = op.forward()
    grads = ops.GradientStore()
    op.backward(grads, do)
    ops.Context.current(q.device).sync()
    want = ref.attn_fwd_bwd(*host, causal=causal)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), [o, op.lse] + [grads.get(t) for t in (q, k, v)], want):
        assert_close(g.cpu().numpy(), w, TOL_F32, f"B {B} H {H} T {T} D {D} {name}")


@pytest.mark.parametrize("M,N,K", [(1, 32, 64), (15, 31, 60), (16, 33, 68), (17, 96, 192), (100, 576, 192), (100, 192, 768), (64, 64, 400), (20, 384, 384), (231, 192, 190), (9, 1020, 256)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 1), (0, 0), (1, 1), (1, 0)])
@pytest.mark.parametrize("aligned", [True, False])
def test_f32_gemm_tiles_of_16_rows(M, N, K, a_mn, b_mn, aligned):
    """Products of few tiles: rows, columns and k that end inside a tile of 16 x 32 or a group's share, clusters, each order, rows on 16-byte boundaries
    and on none; 2e-6 max(1, sqrt(K) / 4) of the largest value, as for the other tiles."""
    from deers_b200 import gpt
    rng = np.random.default_rng(M * 5 + N * 3 + K)
    pad = 0 if aligned else 1

    def operand(rows, cols):
        whole = torch.from_numpy(rng.standard_normal((rows, (cols + 3) // 4 * 4 + pad)).astype(np.float32)).cuda()
        return whole[:, pad:cols + pad]

    a, b = operand(*((K, M) if a_mn else (M, K))), operand(*((K, N) if b_mn else (N, K)))
    out = torch.full((M, (N + 3) // 4 * 4 + 4), float("nan"), device="cuda")
    r = torch.from_numpy(rng.standard_normal((M, (N + 3) // 4 * 4)).astype(np.float32)).cuda()
    gpt.gemm_f32(a, b, bool(a_mn), bool(b_mn), out=out[:, :N])
    want = (a.double().T if a_mn else a.double()) @ (b.double() if b_mn else b.double().T)
    bound = 2e-6 * max(1.0, K ** 0.5 / 4) * want.abs().max().item()
    assert (out[:, :N].double() - want).abs().max().item() <= bound and out[:, N:].isnan().all()
    from deers_b200 import _lib
    got = gpt.gemm_f32(a, b, bool(a_mn), bool(b_mn), epilogue=_lib.EPI_ADD, residual=r[:, :N])
    assert (got.double() - want - r[:, :N].double()).abs().max().item() <= bound + 1e-6


@pytest.mark.parametrize("C", [4, 124, 128, 132, 192, 252, 256, 260])
@pytest.mark.parametrize("rows", [1, 9, 20000])
def test_rmsnorm_backward_of_short_rows(rows, C):
    """Rows of up to 256, whose loads all go out at once, and the next longer ones; fewer rows than a block's warps and more than a grid's.  A lane
    adds C / 32 products, five sums of lanes and a few roundings follow: (C / 32 + 12) 2^-24 for the dot product, half as much for the norm, whose third power
    stands in the second term: 3 (C / 32 + 12) 2^-24 of the terms' magnitudes."""
    from deers_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    x, dy = (torch.randn((rows, C), device="cuda", generator=g) for _ in range(2))
    op = ops.RMSNorm.new(x, 1e-5)
    op.forward()
    grads = ops.GradientStore()
    op.backward(grads, dy)
    dx = grads.get(op.dependencies()[0])
    xd, gd = x.double(), dy.double()
    r = (xd.square().mean(1, keepdim=True) + 1e-5).rsqrt()
    dot = (xd * gd).sum(1, keepdim=True)
    want = gd * r - xd * dot * r ** 3 / C
    terms = (gd * r).abs() + xd.abs() * (xd * gd).abs().sum(1, keepdim=True) * r ** 3 / C
    assert ((dx.double() - want).abs() <= 3 * (C / 32 + 12) * 2.0 ** -24 * terms).all()
