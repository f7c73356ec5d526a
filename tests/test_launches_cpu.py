"""CPU tier: the host side of the launches against a stand-in CUDA runtime (fake_cudart.c): what a failing call leaves behind,
what two host threads do to each other, which grid a problem gets.  Each check runs in a process of its own, this file as the
program, with the stand-in preloaded."""
import ctypes
import os
import shutil
import subprocess
import sys
import threading

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "amd-kernels_b200", "kernels", "libhkb200.so")
HKB_OK, HKB_ERR_CUDA = 0, -5
i64 = ctypes.c_int64
LAUNCH = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_char_p, ctypes.c_uint, ctypes.c_uint, ctypes.c_size_t, ctypes.c_int, ctypes.c_int,
                          ctypes.POINTER(ctypes.c_void_p))
CALL = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_char_p, ctypes.c_int)


class Runtime:
    """The stand-in's side of a check.  on_launch / on_limit / on_call may be replaced; what they return is what the call returns."""
    def __init__(self):
        self.fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
        self.lib = ctypes.CDLL(LIB)
        self.lib.hkb_last_error.restype = self.lib.hkb_last_kernel.restype = ctypes.c_char_p
        self.on_launch = lambda name, grid, smem, args: 0
        self.on_limit = lambda name, value: 0
        self.on_call = lambda name, value: 0
        self._keep = (LAUNCH(lambda n, g, b, s, c, e, a: self.on_launch(n.decode(), g, s, a)),
                      CALL(lambda n, v: self.on_limit(n.decode(), v)), CALL(lambda n, v: self.on_call(n.decode(), v)))
        self.fake.fake_callbacks(*self._keep)

    @staticmethod
    def p(n=1):
        return [ctypes.c_void_p((1 << 30) + (i << 33)) for i in range(n)]

    def quant(self, M=64, K=512):
        return self.lib.hkb_quant_fp8_per_token(*self.p(3), i64(M), i64(K), i64(K), None)

    def pts(self, M, N, K, batch=1):
        return self.lib.hkb_gemm_fp8_pts(*self.p(5), None, i64(batch), i64(M), i64(N), i64(K), None)

    def blockscale(self, M, N, K):
        return self.lib.hkb_gemm_fp8_blockscale(*self.p(5), i64(128), i64(M), i64(N), i64(K), None)

    def mxfp4(self, M, N, K, batch=1):
        return self.lib.hkb_gemm_mxfp4(*self.p(5), i64(batch), i64(M), i64(N), i64(K), None)

    def mxfp4_tc(self, M, N, K, batch=1):
        a, b, c, sa, sb = self.p(5)
        return self.lib.hkb_gemm_mxfp4_tc(a, b, c, sa, 1, sb, 1, i64(batch), i64(M), i64(N), i64(K), None)

    def mxfp4_static(self, M, N, K):
        return self.lib.hkb_gemm_mxfp4_static(*self.p(5), i64(1), i64(M), i64(N), i64(K), None)

    def ptgq(self, M, N, K):
        return self.lib.hkb_gemm_fp8_ptgq(*self.p(4), None, i64(1), i64(M), i64(N), i64(K), None)

    def moe_fp8(self, rows, N, K):
        x, w, y, xs, ws, g, h, o, d = self.p(9)
        return self.lib.hkb_moe_gemm_fp8_blockscale(x, w, y, xs, ws, None, g, h, o, d, i64(rows // 2), i64(rows), i64(8), i64(N), i64(K),
                                                    i64(rows // 128 + 8), i64(2), None)

    def moe_mxfp4(self, rows, N, K):
        a, b, c, sa, sb, w, ids, ex = self.p(8)
        return self.lib.hkb_moe_gemm_mxfp4(a, b, c, sa, sb, None, None, w, ids, ex, i64(rows // 2), i64(rows), i64(8), i64(N), i64(K),
                                           i64(rows), i64(2), 1, None)

    def calls(self):
        """One call per kernel that is launched."""
        return {"quantizer": self.quant, "per-token decode": lambda: self.pts(16, 4096, 1024), "per-token pairs": lambda: self.pts(4096, 8192, 512),
                "per-token 64": lambda: self.pts(512, 1024, 512), "block-scale decode": lambda: self.blockscale(16, 4096, 1024),
                "block-scale 128": lambda: self.blockscale(512, 1024, 512), "block-scale 256": lambda: self.blockscale(4096, 8192, 512),
                "MXFP4 decode": lambda: self.mxfp4(16, 4096, 1024), "MXFP4 128": lambda: self.mxfp4(512, 1024, 512),
                "MXFP4 192": lambda: self.mxfp4_tc(1000, 3080, 512), "MXFP4 pairs": lambda: self.mxfp4(4096, 8192, 512),
                "MXFP4 static": lambda: self.mxfp4_static(256, 512, 512), "in-loop": lambda: self.ptgq(256, 512, 512),
                "MoE FP8": lambda: self.moe_fp8(512, 1024, 512), "MoE MXFP4": lambda: self.moe_mxfp4(512, 1024, 512)}


def check_failed_calls_leave_no_error_pending():
    """A launch, an attribute, an allocation that fails is that call's error and nobody else's: the thread's pending error is taken
    back, so that the next launch -- this library's or another's -- is not reported as failed."""
    rt = Runtime()
    for what, call in rt.calls().items():
        assert call() == HKB_OK, (what, rt.lib.hkb_last_error())
        failed = []

        def fail_at(n):
            seen = [0]

            def hit(name, *_):
                seen[0] += 1
                if seen[0] == n:
                    failed.append(name)
                    return 701
                return 0
            return hit

        for hook in ("on_launch", "on_limit", "on_call"):
            for n in (1, 2, 3):
                rt.lib.hkb_release()                     # scratch is allocated again
                failed.clear()
                setattr(rt, hook, fail_at(n))
                rc = call()
                setattr(rt, hook, lambda *_: 0)
                if not failed:
                    break
                assert rc == HKB_ERR_CUDA, (what, hook, n, rc)
                assert rt.fake.fake_pending() == 0, (what, hook, failed)
                assert rt.quant() == HKB_OK and call() == HKB_OK, (what, hook, failed, rt.lib.hkb_last_error())


def check_two_threads_do_not_take_each_others_shared_memory():
    """The shared-memory limit belongs to the kernel, not to the call: a call of another shape from another thread, coming between
    a call's setting it and its launch, must not make that launch ask for more than the limit allows."""
    rt = Runtime()
    limit, asked, between = {}, {}, []

    def on_limit(name, value):
        limit[name] = value
        if between:
            other = threading.Thread(target=lambda call: inner.append(call()), args=(between.pop(),))
            other.start()
            other.join()
        return 0

    def on_launch(name, grid, smem, args):
        asked.setdefault(name, set()).add(smem)
        return 0 if smem <= limit.get(name, 48 << 10) else 1                     # cudaErrorInvalidValue

    rt.on_limit, rt.on_launch = on_limit, on_launch
    shapes = [(M, N, K) for M in (1, 16, 32) for N, K in [(1024, 1024), (4096, 4096), (14336, 4096), (28672, 8192)]]
    for kind in (rt.pts, rt.blockscale, rt.mxfp4):
        for a in shapes:
            for b in shapes:
                inner = []
                between[:] = [lambda: kind(*b)]
                rc = kind(*a)
                between.clear()
                assert rc == HKB_OK and all(r == HKB_OK for r in inner), (rt.lib.hkb_last_kernel(), a, b, rt.lib.hkb_last_error())
    assert sum(len(v) > 1 for v in asked.values()) >= 3, asked                    # decode kernels whose size depends on the shape


def check_mxfp4_tiles_cover_the_result_once():
    """The row and column tile counts that an MXFP4 kernel walks are those of its own tile, and no cluster or block is left
    without one: a count for another width leaves columns out or walks tiles that lie wholly past N."""
    rt = Runtime()
    tiles = {"gemm_mxfp4_pair_kernel<256x192>": (256, 192, 2), "gemm_mxfp4_kernel<192>": (128, 192, 1), "gemm_mxfp4_kernel<128>": (128, 128, 1)}
    launched = []

    def on_launch(name, grid, smem, args):
        if "gemm_mxfp4" in name:
            p = 4 if "pair" in name else 2                                       # behind the tensor maps: M, N, K, batch, m_blks, n_blks
            launched.append((grid, ctypes.cast(args[p], ctypes.POINTER(ctypes.c_int))[:6]))
        return 0

    rt.on_launch = on_launch
    seen = set()
    for batch in (1, 3):
        for M in [100, 129, 300] + list(range(640, 8193, 64 if batch == 1 else 640)):
            for N in [8, 136, 1000] + list(range(1024, 28673, 512 if batch == 1 else 1920)):
                launched.clear()
                assert rt.mxfp4_tc(M, N, 1024, batch) == HKB_OK, rt.lib.hkb_last_error()
                kernel = rt.lib.hkb_last_kernel().decode()
                seen.add(kernel)
                bm, bn, ctas = tiles[kernel]
                (grid, got), = launched
                want = [M, N, 1024, batch, -(-M // bm), -(-N // bn)]
                assert got == want, (kernel, got, want)
                assert grid == ctas * min(148 // ctas, batch * want[4] * want[5]), (kernel, grid, want)
    assert seen == set(tiles), seen


class GemmParams(ctypes.Structure):
    """The FP8 GEMM kernels' parameters (csrc/gemm_fp8.cu) up to the field that is read here."""
    _fields_ = ([(n, ctypes.c_int) for n in "M N K batch m_blks n_blks a_box_rows".split()] + [(n, ctypes.c_void_p) for n in "sa sb bias C".split()] +
                [("gn", ctypes.c_int), ("c_a", ctypes.c_void_p), ("c_b", ctypes.c_void_p), ("ldc", i64), ("peer", ctypes.c_void_p * 7), ("n_peer", ctypes.c_int)] +
                [(n, ctypes.c_void_p) for n in "expt_data expt_hist expt_offs bias_f32 c2".split()] +
                [(n, ctypes.c_int) for n in "sc_s1 sc_s2 sc_s3 group_m split_from".split()])


def check_per_token_pairs_split_a_small_last_wave():
    """What the CTA-pair kernel is told to walk: 256 x 256 tiles over 74 clusters, those of a last wave that fills at most half of
    the clusters as two halves each, everything else whole."""
    rt = Runtime()
    launched = []

    def on_launch(name, grid, smem, args):
        p = GemmParams.from_address(args[2])
        launched.append((grid, p.M, p.N, p.K, p.batch, p.m_blks, p.n_blks, p.group_m, p.split_from))
        return 0

    rt.on_launch = on_launch
    split = whole = 0
    for batch, M, N in [(8, 512, 4096), (2, 1290, 5000), (1, 2300, 6408)] + [(1, M, N) for M in range(1024, 8193, 640) for N in range(2048, 16385, 1024)]:
        launched.clear()
        assert rt.pts(M, N, 256, batch) == HKB_OK, rt.lib.hkb_last_error()
        if rt.lib.hkb_last_kernel() != b"gemm_fp8_kernel<256,pts,pair>":
            continue
        mb, nb = -(-M // 256), -(-N // 256)
        tiles = batch * mb * nb
        tail = tiles % 74 if tiles > 74 else 0
        want = tiles - tail if 0 < tail <= 37 else tiles
        assert launched == [(2 * min(74, tiles), M, N, 256, batch, mb, nb, 8, want)], (launched, want)
        split, whole = split + (want < tiles), whole + (want == tiles)
    assert split > 20 and whole > 20, (split, whole)


def _run(check, tmp_path):
    import pytest
    inc = "/usr/local/cuda/include"
    gcc = shutil.which("gcc")
    if gcc is None or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no C compiler or CUDA runtime headers")
    so = str(tmp_path / "fake_cudart.so")
    src = os.path.join(ROOT, "tests", "fake_cudart.c")
    subprocess.run([gcc, "-std=gnu11", "-O1", "-shared", "-fPIC", "-I", inc, src, "-o", so], check=True, capture_output=True, text=True)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), check], env={**os.environ, "LD_PRELOAD": so}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_failed_calls_leave_no_error_pending(tmp_path):
    _run("check_failed_calls_leave_no_error_pending", tmp_path)


def test_two_threads_do_not_take_each_others_shared_memory(tmp_path):
    _run("check_two_threads_do_not_take_each_others_shared_memory", tmp_path)


def test_mxfp4_tiles_cover_the_result_once(tmp_path):
    _run("check_mxfp4_tiles_cover_the_result_once", tmp_path)


def test_per_token_pairs_split_a_small_last_wave(tmp_path):
    _run("check_per_token_pairs_split_a_small_last_wave", tmp_path)


if __name__ == "__main__":
    globals()[sys.argv[1]]()
