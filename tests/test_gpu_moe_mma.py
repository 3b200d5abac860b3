"""GPU parity of the routed experts over many rows (the prompt path's jobs of up to 64 rows, tcgen05 tensor cores)
against the CPU oracle through the C ABI: the f16 weights bit for bit (read back through one-hot rows), the sums to a
stated bound on fp32 summation error, SwiGLU to f16 bit for bit."""
import ctypes as C

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu


def _f16_bits(a):
    return np.ascontiguousarray(a.astype(np.float16)).view(np.uint16)


def _run(entry, experts, jobs, x16, nout):
    import torch

    from sfnx_b200 import lib as L
    from tests import gpu_util as G

    st = L.stream()
    dj = G.dev(jobs.view(np.uint8).reshape(-1))
    nj = G.dev(np.array([len(jobs), 0], np.int32))
    dx = G.dev(x16)
    out = torch.full((nout, experts.nrows), float("nan"), device="cuda")
    L.call(entry, C.byref(experts), dj.data_ptr(), nj.data_ptr(), len(jobs) + 3, dx.data_ptr(), out.data_ptr(), st)   # spare grid rows do nothing
    G.sync()
    assert L.load().fnx_device_fault() == 0
    return G.host(out)


def _close(got, ref, mag, n):
    """fp32 sums of exact products in an unstated order, one partial sum per 16 columns: each step may lose one fp32 unit
    in the last place of the running magnitude, so |got - ref| <= (n / 16 + 8) 2^-23 sum|products|."""
    bound = (n / 16 + 8) * 2.0 ** -23 * mag + 1e-30
    err = np.abs(got.astype(np.float64) - ref)
    assert np.isfinite(got).all()
    assert (err <= bound).all(), (float((err / bound).max()), float(err.max()))


def _experts(w, which):
    from tests import gpu_util as G

    n, ffs = w["n"], w["ffs"]
    if w.get("experts") == "q8_0":
        return G.experts_q8(w["gu_q8"], 2 * ffs, n) if which == "gu" else G.experts_q8(w["dn_q8"], n, ffs)
    return G.experts_q4k(w["gu_q4k"], 2 * ffs, n) if which == "gu" else G.experts_q6p(w["dn_planes"], n, ffs)


def _weights16(w, which):
    """The oracle's f16 weights [experts * rows][cols]."""
    from oracle import binding as O

    n, ffs, nexp = w["n"], w["ffs"], w["nexp"]
    if w.get("experts") == "q8_0":
        q, d = w["gu_q8"] if which == "gu" else w["dn_q8"]
        return O.mma_weights_q8(q, d)
    if which == "gu":
        return O.mma_weights_q4k(w["gu_q4k"], nexp * 2 * ffs, n)
    return O.mma_weights_q6p(w["dn_planes"], nexp * n, ffs)


@pytest.mark.parametrize("kind", ["q4k", "q8_0"])
def test_f16_weights_bit_exact_through_one_hot_rows(kind):
    """Row s of a job is the unit vector of column 64 j + s: the job's output is 64 columns of the expert's f16 weights,
    each sum a single non-zero product, so the dequantisation is read back bit for bit."""
    n, ffs, nexp = 512, 256, 3
    w = (cases.moe_weights if kind == "q4k" else cases.moe_weights_q8)(n=n, nexp=nexp, ffs=ffs, seed=31)
    from oracle import binding as O

    for which, cols, rows in (("gu", n, 2 * ffs), ("dn", ffs, n)):
        x = np.zeros((cols, cols), np.float16)
        x[np.arange(cols), np.arange(cols)] = 1
        jobs = np.zeros(nexp * cols // 64, O.BIGJOB_DTYPE)
        for e in range(nexp):
            for j in range(cols // 64):
                jb = jobs[e * (cols // 64) + j]
                jb["w"], jb["n"] = e, 64
                jb["y"][:] = np.arange(64) + 64 * j
                jb["out"][:] = e * cols + jb["y"]
        ex, keep = _experts(w, which)
        got = _run("fnx_moe_gate_up_mma" if which == "gu" else "fnx_moe_down_mma", ex, jobs, x.view(np.uint16), nexp * cols)
        ref = _weights16(w, which).view(np.float16).reshape(nexp, rows, cols).transpose(0, 2, 1).reshape(nexp * cols, rows)
        assert np.array_equal(got.astype(np.float32).view(np.uint32), ref.astype(np.float32).view(np.uint32)), which


@pytest.mark.parametrize("kind,n,ffs,nexp,ntok,topk", [("q4k", 512, 256, 8, 150, 4), ("q8_0", 1024, 96, 6, 70, 3), ("q4k", 3072, 768, 4, 150, 2),
                                                      ("q4k", 256, 64, 5, 1, 2), ("q8_0", 256, 64, 2, 330, 2),
                                                      ("q8_0", 256, 32, 3, 40, 2), ("q4k", 256, 32, 3, 40, 2)])
def test_gate_up_swiglu_down(kind, n, ffs, nexp, ntok, topk):
    """gate|up -> SwiGLU -> down over jobs of 1 to 64 rows (ragged job sizes, row tiles past the matrix's last row, FF slice
    96; experts with one, two and six jobs: consecutive jobs of an expert are taken in pairs), each step against the
    oracle fed with the GPU's previous step."""
    from oracle import binding as O

    w = (cases.moe_weights if kind == "q4k" else cases.moe_weights_q8)(n=n, nexp=nexp, ffs=ffs, seed=32)
    jobs, P = cases.big_jobs(ntok, nexp, topk, seed=33)
    rng = np.random.default_rng(34)
    x16 = _f16_bits(rng.standard_normal((ntok, n)))
    ex, keep = _experts(w, "gu")
    gu = _run("fnx_moe_gate_up_mma", ex, jobs, x16, P)
    ref, mag = O.moe_mma(_weights16(w, "gu"), jobs, len(jobs), x16, 2 * ffs, P)
    _close(gu, ref, mag, n)

    import torch

    from sfnx_b200 import lib as L
    from tests import gpu_util as G

    dgu, h16 = G.dev(gu), torch.zeros((P, ffs), dtype=torch.int16, device="cuda")
    L.call("fnx_swiglu_h16", dgu.data_ptr(), ffs, P, h16.data_ptr(), L.stream())
    G.sync()
    h = G.host(h16, np.uint16)
    assert np.array_equal(h, O.swiglu_h16(gu, ffs)), "h = f16(silu(gate) * up)"

    dn_jobs = jobs.copy()
    for jb in dn_jobs:   # the down jobs read the pairs' h rows
        jb["y"][:jb["n"]] = jb["out"][:jb["n"]]
    ex, keep2 = _experts(w, "dn")
    part = _run("fnx_moe_down_mma", ex, dn_jobs, h, P)
    ref, mag = O.moe_mma(_weights16(w, "dn"), dn_jobs, len(dn_jobs), h, n, P)
    _close(part, ref, mag, ffs)


@pytest.mark.parametrize("njobs,nexp", [(5000, 7), (2049, 1), (2048, 3), (600, 600)])
def test_many_jobs(njobs, nexp):
    """More jobs than are listed at a time (2048): runs of one expert's jobs of every parity, some across the lists' ends, one
    expert for all, an expert a job; a tile's two jobs with one to three rows each."""
    from oracle import binding as O

    n, rows = 256, 128
    rng = np.random.default_rng(njobs)
    w = cases.moe_weights_q8(n=n, nexp=nexp, ffs=rows // 2, seed=41)
    lens = rng.integers(1, 3 if nexp > 500 else 40, njobs)
    run = np.arange(njobs) if nexp == njobs else np.repeat(np.arange(njobs), lens)[:njobs]
    jobs = np.zeros(njobs, O.BIGJOB_DTYPE)
    P = 0
    x16 = _f16_bits(rng.standard_normal((97, n)))
    for j in range(njobs):
        k = int(rng.integers(1, 4))
        jobs[j]["w"], jobs[j]["n"] = run[j] % nexp, k
        jobs[j]["y"][:k], jobs[j]["out"][:k] = rng.integers(0, 97, k), np.arange(P, P + k)
        P += k
    ex, keep = _experts(w, "gu")
    got = _run("fnx_moe_gate_up_mma", ex, jobs, x16, P)
    ref, mag = O.moe_mma(_weights16(w, "gu"), jobs, njobs, x16, rows, P)
    _close(got, ref, mag, n)


@pytest.mark.parametrize("cap,count", [(1, 6), (4, 6), (5, 2048), (2047, 5000), (2049, 5000)])
def test_no_job_past_the_capacity(cap, count):
    """A count on the device above the caller's njobs_cap: the jobs up to it are done, those past it (valid ones here, of the
    same expert as the last) are neither done nor taken as a partner."""
    import torch

    from oracle import binding as O
    from sfnx_b200 import lib as L
    from tests import gpu_util as G

    n, rows = 256, 128
    w = cases.moe_weights_q8(n=n, nexp=3, ffs=rows // 2, seed=42)
    jobs = np.zeros(count, O.BIGJOB_DTYPE)
    jobs["w"], jobs["n"] = np.arange(count) // 3 % 3, 1   # runs of three jobs an expert
    jobs["y"][:, 0], jobs["out"][:, 0] = np.arange(count) % 97, np.arange(count)
    x16 = _f16_bits(np.random.default_rng(43).standard_normal((97, n)))
    ex, keep = _experts(w, "gu")
    dj, nj, dx = G.dev(jobs.view(np.uint8).reshape(-1)), G.dev(np.array([count, 0], np.int32)), G.dev(x16)
    out = torch.full((count, rows), float("nan"), device="cuda")
    L.call("fnx_moe_gate_up_mma", C.byref(ex), dj.data_ptr(), nj.data_ptr(), cap, dx.data_ptr(), out.data_ptr(), L.stream())
    G.sync()
    assert L.load().fnx_device_fault() == 0
    got = G.host(out)
    ref, mag = O.moe_mma(_weights16(w, "gu"), jobs[:cap], cap, x16, rows, count)
    _close(got[:cap], ref[:cap], mag[:cap], n)
    assert np.isnan(got[cap:]).all()


@pytest.mark.parametrize("kind,n,ffs", [("q4k", 768, 288), ("q4k", 256, 288), ("q8_0", 800, 288), ("q8_0", 736, 96)])
def test_many_tiles_a_block(kind, n, ffs):
    """Three and more tiles for every block of the persistent kernel, gate|up and down: matrices of two and a half to four tiles
    of rows, jobs of 1 to 64 rows alone and in pairs (64 + 64 among them), one to thirteen steps with and without a last one
    of 32 columns.  What is carried from tile to tile (the raw ring, the scales asked for ahead, the two results in tensor
    memory) shows in the sums."""
    from oracle import binding as O

    nexp, sizes = 7, ([1], [17], [64], [2], [64, 64], [3, 9], [5])
    w = (cases.moe_weights if kind == "q4k" else cases.moe_weights_q8)(n=n, nexp=nexp, ffs=ffs, seed=44)
    rng = np.random.default_rng(45)
    for which, rows, cols in (("gu", 2 * ffs, n), ("dn", n, ffs)):
        tiles = (rows + 255) // 256
        pairs = (3 * 160 + tiles - 1) // tiles
        take = [(g % nexp, k) for g in range(pairs) for k in sizes[g % len(sizes)]]
        jobs, P = np.zeros(len(take), O.BIGJOB_DTYPE), 0
        x16 = _f16_bits(rng.standard_normal((131, cols)))
        for jb, (e, k) in zip(jobs, take):
            jb["w"], jb["n"] = e, k
            jb["y"][:k], jb["out"][:k] = rng.integers(0, 131, k), np.arange(P, P + k)
            P += k
        ex, keep = _experts(w, which)
        got = _run("fnx_moe_gate_up_mma" if which == "gu" else "fnx_moe_down_mma", ex, jobs, x16, P)
        ref, mag = O.moe_mma(_weights16(w, which), jobs, len(jobs), x16, rows, P)
        _close(got, ref, mag, cols)


@pytest.mark.parametrize("P,ffs,off", [(1, 5, 0), (7, 33, 0), (40, 12, 0), (3, 64, 1), (1, 8, 2), (513, 96, 3)])
def test_swiglu_of_any_width_and_address(P, ffs, off):
    """Widths that are no whole 16-byte pieces and arrays that begin off a 16-byte boundary (the value-a-thread kernel)."""
    import torch

    from oracle import binding as O
    from sfnx_b200 import lib as L
    from tests import gpu_util as G

    gu = (3 * np.random.default_rng(ffs).standard_normal((P, 2 * ffs))).astype(np.float32)
    dgu = torch.zeros(off + gu.size, device=G.DEV)
    dgu[off:] = G.dev(gu).reshape(-1)
    h = torch.zeros(off + P * ffs + 1, dtype=torch.int16, device=G.DEV)
    L.call("fnx_swiglu_h16", dgu[off:].data_ptr(), ffs, P, h[off:].data_ptr(), L.stream())
    G.sync()
    got = G.host(h, np.uint16)
    assert np.array_equal(got[off:off + P * ffs].reshape(P, ffs), O.swiglu_h16(gu, ffs))
    assert not got[:off].any() and got[-1] == 0


@pytest.mark.parametrize("kind,rows,cols", [("q8_0", 100, 32), ("q8_0", 100, 96), ("q8_0", 300, 64), ("q8_0", 1, 32), ("q4k", 100, 256), ("q4k", 64, 512),
                                            ("q6p", 256, 32), ("q6p", 512, 96)])
def test_nothing_is_read_past_the_end_of_memory(kind, rows, cols):
    """Small matrices, jobs and activation rows that end where their mapped memory does: buffers of 12 MB, mappings of their
    own, each with its array in the last bytes."""
    import torch

    from oracle import binding as O
    from sfnx_b200 import lib as L
    from tests import gpu_util as G

    nexp, rng = 4, np.random.default_rng(rows + cols)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    keep = []

    def tail(a):   # the array's bytes at the end of a mapping, on a 16-byte boundary (what is left over lies behind it)
        b = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
        buf = torch.zeros(12 << 20, dtype=torch.uint8, device=G.DEV)
        at = (buf.numel() - b.size) // 16 * 16
        buf[at:at + b.size] = torch.from_numpy(b.copy()).to(G.DEV)
        keep.append(buf)
        return buf.data_ptr() + at

    if kind == "q8_0":
        q = rng.integers(-127, 128, (nexp, rows, cols)).astype(np.int8)
        d = (0.01 * rng.random((nexp, rows, cols // 32)) + 1e-3).astype(np.float16).view(np.uint16)
        ex, w16 = L.Experts(L.Q8_0, rows, cols, tail(q), tail(d), None, None, rows * cols, rows * (cols // 32) * 2), O.mma_weights_q8(q, d)
    elif kind == "q4k":
        w = cases.moe_weights(n=cols, nexp=nexp, ffs=32 * ((rows // 2 + 31) // 32), seed=46)
        blocks = np.ascontiguousarray(w["gu_q4k"].reshape(nexp, -1)[:, :rows * (cols // 256) * 144])
        ex, w16 = L.Experts(L.Q4_K, rows, cols, tail(blocks), None, None, None, blocks.shape[1], 0), O.mma_weights_q4k(blocks, nexp * rows, cols)
    else:
        planes = cases.moe_weights(n=rows, nexp=nexp, ffs=cols, seed=46)["dn_planes"]
        ex, w16 = L.Experts(L.Q6_K, rows, cols, *[tail(p) for p in planes], rows * (cols // 32), 0), O.mma_weights_q6p(planes, nexp * rows, cols)
    n = np.array([1, 40, 64, 3, 64, 17])
    jobs = np.zeros(len(n), O.BIGJOB_DTYPE)
    jobs["w"], jobs["n"] = [0, 1, 2, 2, 3, 3], n
    for j, at in enumerate(np.cumsum(n) - n):
        jobs[j]["y"][:n[j]], jobs[j]["out"][:n[j]] = (np.arange(n[j]) + at) % 71, np.arange(n[j]) + at
    P = int(n.sum())
    x16 = _f16_bits(rng.standard_normal((71, cols)))
    out = torch.full((P, rows), float("nan"), device=G.DEV)
    nj = G.dev(np.array([len(n), 0], np.int32))
    L.call("fnx_moe_gate_up_mma", C.byref(ex), tail(jobs), nj.data_ptr(), len(n), tail(x16), out.data_ptr(), L.stream())
    G.sync()
    assert L.load().fnx_device_fault() == 0
    ref, mag = O.moe_mma(w16, jobs, len(jobs), x16, rows, P)
    _close(G.host(out), ref, mag, cols)
