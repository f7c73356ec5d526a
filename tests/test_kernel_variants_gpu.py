"""GPU tier: the edges of single kernels and of the dispatch rules between them, against the oracle or an exact restatement."""
import ctypes
import os
import threading

import pytest
import torch

from oracle import gemm
from test_gemm_gpu import (DEV, _check, _dev, _fp8_operands, _moe_call, _moe_mxfp4_call, _moe_mxfp4_routing, _mxfp4_operands,
                           _routing, _status_ok)

pytestmark = pytest.mark.gpu


def _tc_layout(sf, batch, rows, K):
    """Row-major e8m0 bytes -> 512-byte atoms (128 rows x 4 bytes, byte (r % 32) * 16 + (r // 32) * 4 + j), zero-padded."""
    katoms, rblks = (K // 128 + 1) & ~1, 2 * ((rows + 255) // 256) + 2
    full = torch.zeros(batch, rblks * 128, katoms * 4, dtype=torch.uint8, device=sf.device)
    full[:, :rows, : K // 32] = sf.view(batch, rows, K // 32)
    return full.view(batch, rblks, 4, 32, katoms, 4).permute(0, 1, 4, 3, 2, 5).reshape(-1)


@pytest.mark.parametrize("batch,rows,K", [(1, 1, 128), (1, 129, 384), (3, 200, 640), (1, 255, 1024), (2, 128, 1152), (1, 3080, 4224)])
def test_mxfp4_scale_prepass_layout(hk, batch, rows, K):
    """Whole and ragged 128-row blocks, 8-atom chunks and 16-byte row pieces: every byte of the layout."""
    sf = torch.randint(1, 255, (batch * rows, K // 32), generator=torch.Generator().manual_seed(rows), dtype=torch.uint8).to(DEV)
    mod = hk.gemm.afp4wfp4
    out = torch.full((mod.sf_tc_bytes(batch, rows, K),), 0xEE, dtype=torch.uint8, device=DEV)
    mod.sf_to_tc(sf if batch == 1 else sf.view(batch, rows, K // 32), out, K)
    assert torch.equal(out, _tc_layout(sf, batch, rows, K))


@pytest.mark.parametrize("shape,kernel", [((1000, 3080, 384), "gemm_mxfp4_kernel<192>"), ((130, 136, 256), "gemm_mxfp4_kernel<128>"),
                                          ((1100, 1904, 128), "gemm_mxfp4_kernel<128>")])
def test_mxfp4_mul_add_and_tile_width_rule(hk, shape, kernel):
    """Ragged rows and columns in the multiply-add epilogue of both tile widths, at sizes on either side of the width rule."""
    M, N, K = shape
    ac, wc, asc, wsc = _mxfp4_operands(M, N, K)
    g = torch.Generator().manual_seed(3)
    c_a, c_b = torch.randn(M, N, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
    C = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    hk.fused_gemm.afp4wfp4_mul_add.dispatch(_dev(ac), _dev(wc), C, _dev(asc), _dev(wsc), _dev(c_a), _dev(c_b))
    torch.cuda.synchronize()
    assert hk.last_kernel() == kernel
    _status_ok()
    _check(C, gemm.mul_add(gemm.gemm_mxfp4(ac, wc, asc, wsc), c_a, c_b), f"mxfp4 mul_add {shape}")


@pytest.mark.parametrize("batch,M,N,mul_add", [(1, 3456, 4096, False), (1, 3400, 4096, True), (3, 1152, 4096, False)])
def test_mxfp4_pairs_where_one_cta_tiles_would_be_narrow(hk, batch, M, N, mul_add):
    """CTA pairs at sizes for which the width rule of the one-CTA kernels says 128: the pairs walk their own 192-wide tiles."""
    K = 384
    ac, wc, asc, wsc = _mxfp4_operands(M, N, K, batch=batch)
    C = torch.full((batch, M, N) if batch > 1 else (M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    if mul_add:
        g = torch.Generator().manual_seed(3)
        c_a, c_b = torch.randn(M, N, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
        hk.fused_gemm.afp4wfp4_mul_add.dispatch(_dev(ac), _dev(wc), C, _dev(asc), _dev(wsc), _dev(c_a), _dev(c_b))
        ref = gemm.mul_add(gemm.gemm_mxfp4(ac, wc, asc, wsc), c_a, c_b)
    elif batch > 1:
        hk.batched_gemm.afp4wfp4.dispatch(_dev(ac), _dev(wc), C, _dev(asc), _dev(wsc))
        ref = [gemm.gemm_mxfp4(ac[b], wc[b], asc[b], wsc[b]) for b in range(batch)]
    else:
        hk.gemm.afp4wfp4.dispatch(_dev(ac), _dev(wc), C, _dev(asc), _dev(wsc))
        ref = gemm.gemm_mxfp4(ac, wc, asc, wsc)
    torch.cuda.synchronize()
    assert hk.last_kernel() == "gemm_mxfp4_pair_kernel<256x192>"
    _status_ok()
    for c, r in zip(C, ref) if batch > 1 else [(C, ref)]:
        _check(c, r, f"mxfp4 pairs {batch}x{M}x{N}")


@pytest.mark.parametrize("shape", [(1, 16, 128), (7, 2000, 384), (16, 10064, 256), (33, 17600, 128), (64, 9488, 1152), (64, 36000, 256)])
def test_mxfp4_skinny_kernel(hk, shape):
    """Tile widths of 1 to 15 units, one and two rounds, an odd number of K atoms, both layouts of either scale array."""
    M, N, K = shape
    ac, wc, asc, wsc = _mxfp4_operands(M, N, K)
    ref = gemm.gemm_mxfp4(ac, wc, asc, wsc)
    mod = hk.gemm.afp4wfp4
    a, w, sa, sw = (_dev(v) for v in (ac, wc, asc, wsc))
    a_tc = torch.full((mod.sf_tc_bytes(1, M, K),), 0xFF, dtype=torch.uint8, device=DEV)
    w_tc = torch.full((mod.sf_tc_bytes(1, N, K),), 0xFF, dtype=torch.uint8, device=DEV)
    mod.sf_to_tc(sa, a_tc, K)
    mod.sf_to_tc(sw, w_tc, K)
    for a_is_tc, b_is_tc in [(False, False), (True, True), (False, True), (True, False)]:
        C = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        mod.dispatch_tc(a, w, C, a_tc if a_is_tc else sa, w_tc if b_is_tc else sw, a_is_tc, b_is_tc)
        torch.cuda.synchronize()
        wins = N >= 32 * torch.cuda.get_device_properties(0).multi_processor_count or not (a_is_tc and b_is_tc)
        assert hk.last_kernel() == ("gemm_mxfp4_skinny_kernel" if wins else "gemm_mxfp4_kernel<128>")
        _status_ok()
        _check(C, ref, f"mxfp4 skinny {shape} {a_is_tc} {b_is_tc}")
    g = torch.Generator().manual_seed(3)
    c_a, c_b = torch.randn(M, N, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
    hk.fused_gemm.afp4wfp4_mul_add.dispatch(a, w, C, sa, sw, _dev(c_a), _dev(c_b))
    torch.cuda.synchronize()
    _check(C, gemm.mul_add(ref, c_a, c_b), f"mxfp4 skinny mul_add {shape}")


@pytest.mark.parametrize("shape", [(1, 128, 128), (16, 2560, 640), (17, 14336, 1152), (32, 19072, 256), (8, 4096, 2048), (32, 40960, 128)])
def test_blockscale_skinny_kernel(hk, shape):
    """Tile heights of 1 to 8 units, one to three rounds, tiles across two scale groups, partial scale chunks and an odd number
    of K blocks, both token widths; also bit-equal to the large kernel (whose result for rows 0..M of a taller A is the same sum in the same order)."""
    M, N, K = shape
    g = torch.Generator().manual_seed(M)
    A = torch.randint(0, 255, (128, K), generator=g, dtype=torch.uint8)
    B = torch.randint(0, 255, (N, K), generator=g, dtype=torch.uint8)
    for t in (A, B):
        t[(t & 0x7F) > 0x6F] = 0x38                                  # no NaN, magnitudes up to 120
    sa = torch.rand(128, K // 128, generator=g) * 0.1 + 0.01
    sb = torch.rand(K // 128, N // 128, generator=g) * 0.1 + 0.01
    c_a, c_b = torch.randn(128, N, generator=g).bfloat16(), torch.randn(128, N, generator=g).bfloat16()
    a, b, sad, sbd, ca, cb = (t.to(DEV) for t in (A, B, sa, sb, c_a, c_b))
    big, big_ma = (torch.empty(128, N, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    C, C_ma = (torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    hk.gemm.a8w8_blockscale.dispatch(a, b, big, sad, sbd)
    hk.fused_gemm.a8w8_blockscale_mul_add.dispatch(a, b, big_ma, sad, sbd, ca, cb)
    hk.gemm.a8w8_blockscale.dispatch(a[:M], b, C, sad[:M], sbd)
    assert hk.last_kernel() == "gemm_fp8_blockscale_skinny_kernel"
    hk.fused_gemm.a8w8_blockscale_mul_add.dispatch(a[:M], b, C_ma, sad[:M], sbd, ca[:M], cb[:M])
    torch.cuda.synchronize()
    _status_ok()
    _check(C, gemm.gemm_fp8_blockscale(A[:M].numpy(), B.numpy(), sa[:M], sb), f"blockscale skinny {shape}")
    assert torch.equal(C, big[:M]) and torch.equal(C_ma, big_ma[:M])


@pytest.mark.parametrize("kind,M,N", [("blockscale", 1, 128), ("blockscale", 9, 2560), ("blockscale", 32, 19072), ("blockscale", 200, 512),
                                      ("mxfp4", 5, 2560), ("mxfp4", 64, 36000), ("mxfp4", 300, 520), ("mxfp4", 2400, 3072)])
def test_mul_add_in_place(hk, kind, M, N):
    """C may be c_a or c_b itself: both are read ahead of the stores, each element by the thread that then writes it."""
    K = 256
    g = torch.Generator().manual_seed(5)
    if kind == "mxfp4":
        ops = [_dev(v) for v in _mxfp4_operands(M, N, K)]
        dispatch = hk.fused_gemm.afp4wfp4_mul_add.dispatch
    else:
        aq, bq, _, _ = _fp8_operands(M, N, K)
        ops = [_dev(aq), _dev(bq), (torch.rand(M, K // 128, generator=g) * 0.1 + 0.01).to(DEV), (torch.rand(K // 128, N // 128, generator=g) * 0.1 + 0.01).to(DEV)]
        dispatch = hk.fused_gemm.a8w8_blockscale_mul_add.dispatch
    c_a, c_b = (torch.randn(M, N, generator=g).bfloat16().to(DEV) for _ in range(2))
    want, in_a, in_b = torch.empty_like(c_a), c_a.clone(), c_b.clone()
    for C, a, b in [(want, c_a, c_b), (in_a, in_a, c_b), (in_b, c_a, in_b)]:
        dispatch(ops[0], ops[1], C, ops[2], ops[3], a, b)
    torch.cuda.synchronize()
    _status_ok()
    assert torch.equal(in_a, want) and torch.equal(in_b, want) and not torch.equal(want, c_b)


@pytest.mark.parametrize("shape", [(1, 128, 128), (17, 2560, 640), (32, 14336, 256)])
def test_blockscale_skinny_pitched_result(hk, shape):
    """One destination with a row pitch: the column slab of a wider matrix, nothing outside it touched."""
    M, N, K = shape
    aq, bq, _, _ = _fp8_operands(M, N, K, seed=51)
    g = torch.Generator().manual_seed(7)
    sa = torch.rand(M, K // 128, generator=g) * 0.1 + 0.01
    sb = torch.rand(K // 128, N // 128, generator=g) * 0.1 + 0.01
    a, b, sad, sbd = _dev(aq), _dev(bq), sa.to(DEV), sb.to(DEV)
    plain = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    hk.gemm.a8w8_blockscale.dispatch(a, b, plain, sad, sbd)
    ldc, col0 = 2 * N + 48, N + 32
    out = torch.full((M + 1, ldc), 7.0, dtype=torch.bfloat16, device=DEV)
    hk.gemm.a8w8_blockscale.dispatch_scatter(a, b, [out.data_ptr() + col0 * 2], ldc, sad, sbd)
    assert hk.last_kernel() == "gemm_fp8_blockscale_skinny_kernel"
    torch.cuda.synchronize()
    _status_ok()
    _check(plain, gemm.gemm_fp8_blockscale(aq, bq, sa, sb), f"blockscale skinny {shape}")
    assert torch.equal(out[:M, col0:col0 + N], plain)
    out[:M, col0:col0 + N] = 7.0
    assert bool((out == 7.0).all())


@pytest.mark.parametrize("kind", ["pts", "blockscale", "mxfp4"])
def test_decode_kernels_from_two_host_threads(hk, kind):
    """Two shapes whose launches need different amounts of shared memory, each called from its own thread on its own stream through
    the C ABI (ctypes lets go of the interpreter's lock): every call is accepted and gives what it gives alone."""
    lib = ctypes.CDLL(os.path.join(os.path.dirname(hk.__file__), "..", "kernels", "libhkb200.so"))
    i64, K = ctypes.c_int64, 1024
    g = torch.Generator().manual_seed(1)
    jobs = []
    for M, N in [(16, 14336), (1, 1024)]:
        bytes_ = lambda *s: torch.randint(0, 0x70, s, generator=g, dtype=torch.uint8).to(DEV)       # noqa: E731, B023
        scale = lambda *s: (torch.rand(*s, generator=g) * 0.1 + 0.01).to(DEV)                        # noqa: E731, B023
        C = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in range(8)]
        if kind == "mxfp4":
            ops, fn, mid = (bytes_(M, K // 2), bytes_(N, K // 2), bytes_(M, K // 32), bytes_(N, K // 32)), lib.hkb_gemm_mxfp4, (i64(1),)
        elif kind == "pts":
            ops, fn, mid = (bytes_(M, K), bytes_(N, K), scale(M), scale(N)), lib.hkb_gemm_fp8_pts, (None, i64(1))
        else:
            ops, fn, mid = (bytes_(M, K), bytes_(N, K), scale(M, K // 128), scale(K // 128, N // 128)), lib.hkb_gemm_fp8_blockscale, (i64(128),)

        def call(c, stream, ops=ops, fn=fn, mid=mid, M=M, N=N):
            a, b, sa, sb = (ctypes.c_void_p(t.data_ptr()) for t in ops)
            return fn(a, b, ctypes.c_void_p(c.data_ptr()), sa, sb, *mid, i64(M), i64(N), i64(K), ctypes.c_void_p(stream.cuda_stream))

        want = torch.empty_like(C[0])
        assert call(want, torch.cuda.current_stream()) == 0
        jobs.append((call, C, want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    codes = [[] for _ in jobs]
    start = threading.Barrier(len(jobs))

    def work(i):
        call, C, _, stream = jobs[i]
        torch.cuda.set_device(0)
        start.wait()
        for n in range(400):
            codes[i].append(call(C[n % len(C)], stream))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    _status_ok()
    assert codes == [[0] * 400] * len(jobs)
    for _, C, want, _ in jobs:
        assert want.abs().max() > 0 and all(torch.equal(c, want) for c in C)


def test_shim_reads_tensors_parameters_and_subclasses_alike(hk):
    """Plain tensors and Parameters go through the native reads, subclasses through the general ones: same results, same
    refusals, on the current stream of the tensors' device."""
    class Sub(torch.Tensor):
        pass

    x = torch.randn(40, 256, generator=torch.Generator().manual_seed(1)).bfloat16().to(DEV)
    want, ws = torch.empty(40, 256, dtype=torch.uint8, device=DEV), torch.empty(40, 1, device=DEV)
    hk.per_token_quant_fwd(x, want, ws)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for wrap in (lambda t: t, lambda t: torch.nn.Parameter(t, requires_grad=False), lambda t: t.as_subclass(Sub)):
        q, s = torch.zeros_like(want), torch.zeros_like(ws)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(1000000)                # a launch on another stream would overtake this and the zeros below
            q.zero_()
            hk.per_token_quant_fwd(wrap(x), wrap(q), wrap(s))
        side.synchronize()
        assert torch.equal(q, want) and torch.equal(s, ws)
        with pytest.raises(RuntimeError, match="contiguous"):
            hk.per_token_quant_fwd(wrap(x.T), wrap(q), wrap(s))
        with pytest.raises(RuntimeError, match="dtype"):
            hk.per_token_quant_fwd(wrap(x.half()), wrap(q), wrap(s))
        with pytest.raises(RuntimeError, match="CUDA"):
            hk.per_token_quant_fwd(wrap(x.cpu()), wrap(q), wrap(s))


@pytest.mark.parametrize("batch,M,N,K,with_bias", [(8, 512, 4096, 128, True), (1, 2300, 6408, 256, False), (2, 1290, 5000, 384, True)])
def test_per_token_pairs_split_last_wave(hk, batch, M, N, K, with_bias):
    """256 x 256 tiles whose last wave is mostly empty and walked as halves (that they are is shown on the CPU, test_launches_cpu.py);
    rows, columns and halves past the edges."""
    tiles, clusters = batch * -(-M // 256) * -(-N // 256), torch.cuda.get_device_properties(0).multi_processor_count // 2
    if not (tiles > clusters and 0 < 2 * (tiles % clusters) <= clusters):
        pytest.skip(f"{tiles} tiles on {clusters} clusters leave no small last wave")
    aq, bq, sa, sb = _fp8_operands(M, N, K, batch)
    bias = torch.randn(batch, N, generator=torch.Generator().manual_seed(2)).bfloat16() if with_bias else None
    C = torch.full((batch, M, N) if batch > 1 else (M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    if batch > 1:
        hk.batched_gemm.a8w8.dispatch(_dev(aq), _dev(bq), _dev(sa), _dev(sb), C, None if bias is None else _dev(bias))
    else:
        hk.gemm.a8w8_per_token.dispatch(_dev(aq), _dev(bq), C, _dev(sa), _dev(sb))
    torch.cuda.synchronize()
    assert hk.last_kernel() == "gemm_fp8_kernel<256,pts,pair>"
    _status_ok()
    _check(C, gemm.gemm_fp8_per_token(aq, bq, sa, sb, bias), f"per-token pairs {batch}x{M}x{N}x{K}")


def _chained_layers(hk, M, N, K, g):
    """Layers as (quantize(x, operands), new operands, gemm(operands, C), C's shape), weights quantized."""
    E, N_moe = 4, 1024
    mod = hk.gemm.afp4wfp4
    u8 = lambda *s: torch.zeros(*s, dtype=torch.uint8, device=DEV)      # noqa: E731
    f32 = lambda *s: torch.zeros(*s, device=DEV)                         # noqa: E731
    w = (torch.randn(N, K, generator=g) * 0.02).bfloat16().to(DEV)
    wq, ws, bq, bs, fq, fs, ft = u8(N, K), f32(N, 1), u8(N, K), f32(K // 128, N // 128), u8(N, K // 2), u8(N, K // 32), u8(mod.sf_tc_bytes(1, N, K))
    hk.per_token_quant_fwd(w, wq, ws)
    hk.weight_quant_128x128(w, bq, bs)
    hk.fused_rmsnorm_mxfp4_quant_fwd(w, None, fq, fs, 1e-6)
    mod.sf_to_tc(fs, ft, K)
    eq, es = u8(E, N_moe, K), f32(E, K // 128, N_moe // 128)
    eq4, es4 = u8(E, N_moe, K // 2), u8(E, N_moe, K // 32)
    for e in range(E):
        we = (torch.randn(N_moe, K, generator=g) * 0.02).bfloat16().to(DEV)
        hk.weight_quant_128x128(we, eq[e], es[e])
        hk.fused_rmsnorm_mxfp4_quant_fwd(we, None, eq4[e], es4[e], 1e-6)
    hist, offs, gather, data = (_dev(v) for v in _routing(M, E, 2, seed=5))
    ids, eids, gate, total = _moe_mxfp4_routing(M, E, 2, seed=6)
    ids, eids, gate, one = _dev(ids), _dev(eids), _dev(gate), torch.ones(1, device=DEV)
    fp8_1x128 = lambda x, o: hk.fused_rmsnorm_fp8_quant_fwd(x, None, *o, 1e-6)      # noqa: E731
    mxfp4 = lambda x, o: hk.fused_rmsnorm_mxfp4_quant_fwd(x, None, *o, 1e-6)        # noqa: E731
    return [
        (lambda x, o: hk.per_token_quant_fwd(x, *o), lambda: (u8(M, K), f32(M, 1)),
         lambda o, C: hk.gemm.a8w8_per_token.dispatch(o[0], wq, C, o[1], ws), (M, N)),
        (fp8_1x128, lambda: (u8(M, K), f32(M, K // 128)), lambda o, C: hk.gemm.a8w8_blockscale.dispatch(o[0], bq, C, o[1], bs), (M, N)),
        (lambda x, o: hk.fused_rmsnorm_mxfp4_quant_tc_fwd(x, None, o[0], None, o[1], 1e-6), lambda: (u8(M, K // 2), u8(mod.sf_tc_bytes(1, M, K))),
         lambda o, C: mod.dispatch_tc(o[0], fq, C, o[1], ft, True, True), (M, N)),
        (mxfp4, lambda: (u8(M, K // 2), u8(M, K // 32)), lambda o, C: mod.dispatch(o[0], fq, C, o[1], fs), (M, N)),
        (fp8_1x128, lambda: (u8(M, K), f32(M, K // 128)),
         lambda o, C: _moe_call(hk, o[0], eq, C, o[1], es, None, gather, hist, offs, data, 2), (2 * M, N_moe)),
        (mxfp4, lambda: (u8(M, K // 2), u8(M, K // 32)),
         lambda o, C: _moe_mxfp4_call(hk, o[0], eq4, C, o[1], es4, one, one.expand(E).contiguous(), gate, ids, eids, total, 2, True), (2 * M, N_moe)),
    ]


@pytest.mark.parametrize("M,N", [(16, 5120), (300, 5120), (300, 25600)])      # the last one takes the CTA-pair kernels
def test_dependent_launches_under_graph_capture(hk, M, N):
    """Quantizers, pre-passes and GEMMs issued without a wait, eagerly and as a captured chain of programmatic launches, give
    what the same calls give one at a time.  Every layer runs for two inputs in a row (the second rewrites the scratch that the first
    one's GEMM reads), and codes, scales and scratch hold another input's values when a chain starts, so a kernel
    that ran ahead of the one before it would show."""
    K = 1024
    layers = _chained_layers(hk, M, N, K, torch.Generator().manual_seed(M))
    x = [torch.zeros(M, K, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    operands = [[new() for _ in x] for _, new, _, _ in layers]
    C = [[torch.zeros(shape, dtype=torch.bfloat16, device=DEV) for _ in x] for _, _, _, shape in layers]

    def chain(wait=lambda: None, quantizers=True):
        for (quantize, _, multiply, _), ops, c in zip(layers, operands, C):
            for i in (1, 0):
                if quantizers:
                    quantize(x[i], ops[i])
                wait()
            for i in (0, 1):
                multiply(ops[i], c[i])
                wait()

    def fill(seed):
        for i in range(2):
            x[i].copy_(torch.randn(M, K, generator=torch.Generator().manual_seed(2 * seed + i)).bfloat16())

    def poison(seed):
        fill(100 + seed)
        chain(torch.cuda.synchronize)
        for c in C:
            for t in c:
                t.fill_(float("nan"))
        fill(seed)
        torch.cuda.synchronize()

    def same(want):
        torch.cuda.synchronize()
        return [torch.equal(t, v) for c, w in zip(C, want) for t, v in zip(c, w)]

    chain(torch.cuda.synchronize)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        chain()                                                  # scratch is kept per stream and has to exist before a capture
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        chain()
    for seed in range(4):
        fill(seed)
        chain(torch.cuda.synchronize)
        want = [[t.clone() for t in c] for c in C]
        assert all(t.abs().max() > 0 and bool(t.isfinite().all()) for w in want for t in w)
        poison(seed)
        chain(quantizers=False)
        assert not any(same(want))                               # what stale operands would give
        poison(seed)
        chain()
        assert all(same(want))
        poison(seed)
        graph.replay()
        assert all(same(want))
    _status_ok()
