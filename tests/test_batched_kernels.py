"""The batched kernels that fold planes or keep operands in registers, at the edges of their tiles, against 64-bit sums."""
import os
import subprocess

import numpy as np
import pytest

import lutgemm_b200 as L
from lutgemm_b200 import _build, synth
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run(kernel, N, K, q, g, bias, m, column_scales=False, ordered=False, kernel32=None):
    """Two calls against 64-bit sums; `kernel` is the one that has to have run them, `kernel32` where fp32 results take another."""
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + K + m, with_bias=bias)
    if column_scales:
        # columns whose scales lie far apart, down to fp16's subnormals and up to its largest values
        s = 2.0 ** np.random.default_rng(m).integers(-18, 18, N)
        alpha = np.clip(alpha * s, 0, 60000.0 / (q + 1)).astype(np.float16).astype(np.float32)
        q_bias = None if q_bias is None else np.clip(q_bias * s, -9000.0, 9000.0).astype(np.float16).astype(np.float32)
    x = synth.activations(m, K, seed=m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    if ordered:
        w.set_ordered(1)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y32 = torch.empty((m, N), dtype=torch.float32, device="cuda")
    y16 = torch.empty((m, N), dtype=torch.float16, device="cuda")
    first = None
    for _ in range(2):                                    # the second call finds the workspace as the first one left it
        L.matmul_f32(y32, xd, w, m)
        assert L.last_launch()[0] == (kernel32 or kernel)
        L.matmul(y16, xd, w, m)
        assert L.last_launch()[0] == kernel
        if ordered:
            assert first is None or torch.equal(first, y32)
            first = y32.clone()
    a16, b16 = alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16)
    ref = oracle.bcq_matmul_f64(x, bW, a16, b16, g)
    # Products are exact, sums are fp32: every addition errs by at most 2^-23 of the largest partial sum, which is at most
    # |x| |scale| summed; 11 times that with the register operand (up to 6, and its offset of up to 5, for a sign).  K / 16
    # additions per pass.  The split operand's weight is off by up to 2^-22 of it.
    per_add = (2 * K / 16 + 64) * 2.0 ** -23
    grow = {True: 11, False: 1}
    unit = grow[(kernel32 or kernel) == "gemm_frag_kernel"] * per_add + 2.0 ** -22
    mag = np.abs(a16.astype(np.float64)).sum(1) + (0 if b16 is None else np.abs(b16.astype(np.float64)))       # [G, N]
    size = np.abs(x.astype(np.float64)).reshape(m, K // g, g).sum(2) @ mag
    bound = unit * size + 1e-30
    err = np.abs(y32.cpu().numpy().astype(np.float64) - ref)
    assert (err <= bound).all(), (err / bound).max()
    # Per column in the 2-norm, where partial sums of terms of either sign are no larger than the whole (1.5: the spread over
    # 64 rows or more).  A split operand without its low half (2e-4 with these weights) is 6 times beyond this.
    if m >= 64 and 512 <= K <= 1152:
        assert (np.linalg.norm(err, axis=0) <= 1.5 * unit * np.linalg.norm(ref, axis=0)).all()
    # one rounding to fp16 on top: half a unit in the last place, at least half the subnormal step
    with np.errstate(over="ignore"):
        lim = (grow[kernel == "gemm_frag_kernel"] * per_add + 2.0 ** -22) * size + 1e-30 + np.maximum(np.abs(ref) * 2.0 ** -11, 2.0 ** -25)
    got = y16.cpu().numpy().astype(np.float64)
    finite = np.abs(ref) + lim < 65504
    assert (np.abs(got - ref)[finite] <= lim[finite] * 1.0001).all()
    w.close()


# 128-column tiles, 64-k blocks, 16-row steps, 128- and 256-row items, one and several scale groups per block, a last block
# of one word (with one and two scale groups to a block), groups wider than what a warp walks in one stride
@pytest.mark.parametrize("N,K,q,g,bias,m", [
    (8, 32, 4, 32, True, 130), (136, 96, 4, 32, True, 140), (264, 160, 3, 32, True, 300), (128, 64, 3, 64, False, 64), (520, 1024, 2, 32, True, 131), (264, 2048, 2, 128, False, 129),
    (264, 576, 1, 64, True, 130), (1000, 1152, 4, 384, True, 257), (2056, 256, 2, 256, True, 300), (512, 512, 1, 128, False, 144),
    (120, 4096, 3, 1024, True, 100), (4096, 160, 4, 32, False, 513)])
def test_split_operand_kernel(N, K, q, g, bias, m):
    _run("gemm_hl_kernel", N, K, q, g, bias, m)


# fp16 results of few rows: narrow weights of any plane count, and two planes with q_bias; values in registers (up to two planes)
# and in the table, ragged last columns and blocks, one and two scale groups to a block
@pytest.mark.parametrize("N,K,q,g,bias,m", [
    (8, 64, 1, 64, False, 9), (136, 576, 1, 64, True, 12), (264, 2048, 2, 64, False, 16), (2048, 1152, 3, 128, False, 11),
    (520, 4096, 4, 128, False, 33), (2056, 320, 2, 64, True, 9), (4104, 1024, 2, 128, True, 31), (4104, 192, 2, 64, False, 64), (24, 128, 2, 128, True, 63)])
def test_split_operand_kernel_few_rows(N, K, q, g, bias, m):
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + K + m, with_bias=bias)
    x = synth.activations(m, K, seed=m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y = torch.empty((m, N), dtype=torch.float16, device="cuda")
    a16, b16 = alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16)
    ref = oracle.bcq_matmul_f64(x, bW, a16, b16, g)
    # as in _run: K / 16 additions per pass, a weight off by up to 2^-22 of it, one rounding to fp16
    mag = np.abs(a16.astype(np.float64)).sum(1) + (0 if b16 is None else np.abs(b16.astype(np.float64)))
    size = np.abs(x.astype(np.float64)).reshape(m, K // g, g).sum(2) @ mag
    lim = ((2 * K / 16 + 64) * 2.0 ** -23 + 2.0 ** -22) * size + np.maximum(np.abs(ref) * 2.0 ** -11, 2.0 ** -25)
    for _ in range(2):
        L.matmul(y, xd, w, m)
        assert L.last_launch()[0] == "gemm_hl_kernel"
        assert (np.abs(y.cpu().numpy().astype(np.float64) - ref) <= lim * 1.0001).all()
    w.close()


@pytest.mark.parametrize("N,K,q,g,bias,m", [(28672, 1024, 2, 64, True, 16), (12288, 1024, 2, 128, False, 64), (4096, 1024, 1, 64, True, 80),
                                            (11008, 4096, 2, 64, True, 40), (2048, 4096, 2, 128, False, 24)])
def test_split_operand_kernel_few_rows_are_rounded_as_the_plane_kernels(N, K, q, g, bias, m):
    """fp16 results of few rows come from sums as good as the plane kernel's: no more of them, beyond the spread of such a count,
    lie on the wrong side of a rounding than of that kernel's sums, which matmul_f32 gives."""
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + m, with_bias=bias)
    x = synth.activations(m, K, seed=m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y16, y32 = (torch.empty((m, N), dtype=t, device="cuda") for t in (torch.float16, torch.float32))
    L.matmul(y16, xd, w, m)
    assert L.last_launch()[0] == "gemm_hl_kernel"
    L.matmul_f32(y32, xd, w, m)
    assert L.last_launch()[0] == "gemm_tc_kernel"
    ref = oracle.bcq_matmul_f64(x, bW, alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16), g).astype(np.float16)
    off, off_plane = (y16.cpu().numpy() != ref).sum(), (y32.cpu().numpy().astype(np.float16) != ref).sum()
    assert off_plane > 50
    assert off <= off_plane + 4 * np.sqrt(off_plane)
    w.close()


@pytest.mark.parametrize("q,bias,m", [(4, True, 40), (2, False, 150), (1, False, 200), (3, True, 256)])
def test_split_operand_kernel_scales_far_apart(q, bias, m):
    _run("gemm_hl_kernel", 264, 1024, q, 128, bias, m, column_scales=True)


def test_split_operand_kernel_ordered_is_reproducible_and_right():
    _run("gemm_hl_kernel", 264, 2048, 4, 128, True, 140, ordered=True)


# narrow groups up to 128 rows, where a block of 64 k holds several scale groups
@pytest.mark.parametrize("N,K,q,g,bias,m", [(8, 32, 4, 32, True, 17), (136, 96, 4, 32, True, 31), (264, 512, 2, 32, False, 4)])
def test_plane_kernel_narrow_groups(N, K, q, g, bias, m):
    _run("gemm_tc_kernel", N, K, q, g, bias, m)


# 32-column units with ragged last quads and tiles, one to 8 planes, the three kinds of scale group, words beyond K, one and
# two tiles of 8 rows, one and several k-ranges; the last two go 16 rows at a time
@pytest.mark.parametrize("N,K,q,g,bias,m", [
    (4, 32, 1, 32, False, 3), (12, 96, 2, 32, True, 4), (100, 160, 3, 160, False, 5), (36, 4128, 3, 96, True, 3),
    (33 * 4, 1024, 4, 128, True, 8), (5000, 256, 2, 64, False, 7), (264, 8192, 3, 512, False, 4), (40, 2048, 8, 128, True, 6),
    (64, 20480, 5, 64, True, 4), (2052, 4128, 3, 96, False, 16), (20, 384, 7, 192, True, 7), (28, 640, 2, 32, False, 35)])
def test_register_operand_kernel(N, K, q, g, bias, m):
    _run("gemm_frag_kernel", N, K, q, g, bias, m)


# one to four planes have kernels of their own: a last tile of one quad, a last step of two words, several tiles and steps to a warp
@pytest.mark.parametrize("q", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K,g,bias,m", [(68, 192, 64, True, 4), (5220, 1152, 64, False, 8), (68, 128, 128, False, 5), (9508, 768, 384, True, 4),
                                           (68, 160, 32, True, 8), (5220, 1152, 96, False, 4),
                                           (68, 192, 64, True, 9), (5220, 1152, 64, False, 16), (68, 160, 32, True, 16), (1044, 4128, 96, False, 12),
                                           (132, 128, 128, False, 12), (9508, 2304, 384, True, 16)])
def test_register_operand_kernel_per_plane_count(N, K, q, g, bias, m):
    _run("gemm_frag_kernel", N, K, q, g, bias, m)


# one row of containers that tensor maps cannot describe: columns and K that end inside a stage, groups that begin anywhere in
# a slab, wide ones and several to a lane's words, more stages than the ring holds, one nearly empty slab
@pytest.mark.parametrize("N,K,q,g,bias", [
    (4, 32, 1, 32, True), (260, 544, 3, 32, False), (1020, 1056, 4, 96, True), (516, 2080, 2, 160, False), (1284, 1536, 8, 128, True),
    (9000, 1824, 5, 608, False), (132, 3328, 3, 416, True), (2052, 4128, 2, 1376, False), (20484, 576, 7, 64, True)])
def test_matvec_by_copies(N, K, q, g, bias):
    _run("gemv_reg_kernel", N, K, q, g, bias, 1)
    _run("gemv_reg_kernel", N, K, q, g, bias, 1, ordered=True)


# one row where the slabs do not share out evenly: runs of stages that begin and end between planes, cross into one or several
# slabs, hold a column group twice; ragged last groups and slabs; both alpha forms; a run of one stage
@pytest.mark.parametrize("N,K,q,g,bias", [
    (520, 8224, 5, 32, True), (4096, 28672, 3, 256, False), (20488, 1024, 5, 1024, True), (2048, 30720, 7, 64, True),
    (8192, 20480, 1, 128, True), (256, 153088, 1, 512, True), (1032, 40480, 2, 32, False)])
def test_matvec_in_runs(N, K, q, g, bias):
    _run("gemv_flat_kernel", N, K, q, g, bias, 1)


# An infinite activation among the last three of its eight, whose sign a table entry has no sum of both signs of: an infinity where
# the planes (and the offset) agree in sign, else NaN, wherever a run begins and ends.
@pytest.mark.parametrize("kernel,N,K,q,g,bias", [
    ("gemv_flat_kernel", 4096, 28672, 3, 256, True), ("gemv_flat_kernel", 1032, 40480, 2, 32, True), ("gemv_flat_kernel", 8192, 20480, 2, 128, False),
    ("gemv_tma_kernel", 1032, 4096, 3, 128, True), ("gemv_reg_kernel", 1028, 4128, 2, 96, True)])
def test_matvec_activations_not_finite(kernel, N, K, q, g, bias):
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + K, with_bias=bias)
    alpha = np.maximum(alpha, 2.0 ** -10)                 # 0 * inf would be NaN in every column
    x = synth.activations(1, K, seed=K)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias)
    y = torch.empty((1, N), dtype=torch.float32, device="cuda")
    for k, value in ((K // 2 // 8 * 8 + 6, np.inf), (K - 8 + 5, -np.inf), (7, np.inf)):
        xi = x.copy()
        xi[0, k] = value
        bits = (bW[k // 32] >> np.uint32(k % 32)) & np.uint32(1)                                      # [q, N]
        terms = np.where(bits == 1, 1.0, -1.0) * alpha[k // g].astype(np.float16).astype(np.float64)
        if bias:
            terms = np.concatenate([terms, q_bias[k // g].astype(np.float16).astype(np.float64)[None]])
        with np.errstate(invalid="ignore"):
            ref = (terms * np.float64(value)).sum(0)
        assert 0 < np.isinf(ref).sum() < N
        L.matmul_f32(y, torch.from_numpy(xi.view(np.int16)).cuda().view(torch.float16), w, 1)
        assert L.last_launch()[0] == kernel
        assert np.array_equal(y.cpu().numpy()[0], ref.astype(np.float32), equal_nan=True), k
    w.close()


def test_matvec_in_runs_wherever_shared_memory_begins(tmp_path):
    """The lookups' fixed address is where dynamic shared memory begins; instantiated for another one, the kernel still gives the
    result (tests/cpp/flat_any_base.cu compares both with 64-bit sums)."""
    src, exe = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "flat_any_base.cu"), str(tmp_path / "flat_any_base")
    subprocess.check_call([_build.NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", src, "-o", exe],
                          stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "flat ok" in out.stdout, out.stdout + out.stderr


# two and three rows: fp16 results by the register operand, two up to 64 Mi weights of planes and where one slab of k is enough, else
# by the LUT kernels, as fp32 results are
@pytest.mark.parametrize("N,K,q,g,bias,m,kernel", [
    (72, 128, 1, 64, True, 2, "gemm_frag_kernel"), (4096, 4096, 4, 128, False, 2, "gemm_frag_kernel"), (4104, 4096, 4, 128, False, 2, "gemv_tma2_kernel"),
    (72, 8192, 1, 128, False, 2, "gemv_tma2_kernel"), (72, 192, 2, 32, True, 2, "gemv_tma2_kernel"), (72, 8192, 1, 128, True, 3, "gemm_frag_kernel"),
    (72, 192, 2, 32, True, 3, "gemv_tma_kernel")])
def test_two_and_three_rows(N, K, q, g, bias, m, kernel):
    _run(kernel, N, K, q, g, bias, m, kernel32="gemv_tma2_kernel" if m == 2 else "gemv_tma_kernel")


@pytest.mark.parametrize("N,K,q,bias,m", [(4096, 2048, 4, True, 2), (12288, 2048, 4, False, 3)])
def test_fp32_results_of_two_and_three_rows(N, K, q, bias, m):
    """Sums rounded to nearest.  Table entries, of eight fp16 activations, are all but exact; from there a result goes through 7 + q
    additions of a slab and K / 512 slabs, each off by up to half a unit, 2^-24 of a partial sum no larger than the whole, either
    way: 2^-24 / sqrt(3) in the 2-norm, and the root of their number for all."""
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, 128, seed=N + m, with_bias=bias)
    x = synth.activations(m, K, seed=m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // 128, q_bias).reserve_batch(m)
    y = torch.empty((m, N), dtype=torch.float32, device="cuda")
    L.matmul_f32(y, torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16), w, m)
    ref = oracle.bcq_matmul_f64(x, bW, alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16), 128)
    assert np.linalg.norm(y.cpu().numpy() - ref) <= np.sqrt((7 + q + K / 512) / 3) * 2.0 ** -24 * np.linalg.norm(ref)
    w.close()


# planes of 4 GiB, and a k and groups so long that their product has more than 32 bits; a word or a scale from the wrong place is an
# error of the size of the result
@pytest.mark.parametrize("N,K,q,g,bias,rows", [(65540, 131200, 4, 320, False, (4, 16)), (36, 6291456, 1, 3145728, True, (5, 11)), (36, 6291488, 2, 32, True, (8, 9))])
def test_register_operand_kernel_of_wide_containers(N, K, q, g, bias, rows):
    gen = torch.Generator(device="cuda").manual_seed(N + q)
    bW = torch.randint(-2 ** 31, 2 ** 31, (K // 32, q, N), dtype=torch.int32, device="cuda", generator=gen)
    alpha = torch.rand((K // g, q, N), dtype=torch.float16, device="cuda", generator=gen) * 0.02
    q_bias = torch.rand((K // g, N), dtype=torch.float16, device="cuda", generator=gen) * 0.02 if bias else None
    x = torch.rand((max(rows), K), dtype=torch.float16, device="cuda", generator=gen) - 0.5
    w = L.nQWeight_fp16.from_device(bW, alpha, q_bias, K, N, q, False, K // g).reserve_batch(max(rows))
    cols = torch.tensor([0, 3, 17, N // 2, N - 5, N - 1], device="cuda")
    ref = torch.zeros((max(rows), len(cols)), dtype=torch.float64, device="cuda")
    for i, c in enumerate(cols):
        for b in range(q):
            bits = (bW[:, b, c, None] >> torch.arange(32, device="cuda")) & 1
            ref[:, i] += ((bits.reshape(-1) * 2 - 1) * x.double()).reshape(-1, K // g, g).sum(2) @ alpha[:, b, c].double()
        if bias:
            ref[:, i] += x.double().reshape(-1, K // g, g).sum(2) @ q_bias[:, c].double()
    for m in rows:
        y = torch.full((m, N), float("nan"), device="cuda")
        for _ in range(2):
            L.matmul_f32(y, x, w, m)
            assert L.last_launch()[0] == "gemm_frag_kernel"
            assert torch.linalg.norm(y[:, cols].double() - ref[:m]) <= 1e-3 * torch.linalg.norm(ref[:m])
            assert torch.isfinite(y).all()
    w.close()


# k-ranges cost reductions: no more of them where the longest share stays what it is
@pytest.mark.parametrize("N,K,q,g,bias,m,ranges", [(4100, 4096, 2, 64, True, 16, 2), (12292, 4096, 1, 128, False, 16, 2), (12288, 8192, 3, 64, False, 4, 4)])
def test_register_operand_kernel_k_ranges(N, K, q, g, bias, m, ranges):
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + m, with_bias=bias)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    x, y = torch.zeros((m, K), dtype=torch.float16, device="cuda"), torch.empty((m, N), dtype=torch.float16, device="cuda")
    L.matmul(y, x, w, m)
    name, _, gy = L.last_launch()
    assert name == "gemm_frag_kernel"
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert gy == ranges
    assert not y.any()
    w.close()


@pytest.mark.parametrize("q,g,bias,m", [(4, 128, True, 8), (3, 64, False, 4), (2, 32, True, 5)])
def test_register_operand_kernel_scales_far_apart(q, g, bias, m):
    _run("gemm_frag_kernel", 260, 1024, q, g, bias, m, column_scales=True)


def test_three_rows_without_reserved_scratch_inside_a_capture():
    """A first call of three rows inside a stream capture cannot allocate scratch: a container whose register-operand plan
    has several k-ranges still runs it, one row at a time, and with that kernel once scratch is reserved."""
    N, K, q, g = 516, 8160, 3, 96
    bW, alpha, _ = synth.bcq_layer(N, K, q, g, seed=5)
    x = synth.activations(3, K, seed=6)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y = torch.zeros((3, N), dtype=torch.float32, device="cuda")
    ref = oracle.bcq_matmul_f64(x, bW, alpha.astype(np.float16), None, g)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        L.matmul_f32(y, xd, w, 3)
    assert L.last_launch()[0] == "gemv_reg_kernel"
    graph.replay()
    torch.cuda.synchronize()
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-5 * np.linalg.norm(ref)
    assert w.scratch() == (0, 0, 0)
    w.reserve_batch(3)
    L.matmul_f32(y.zero_(), xd, w, 3)
    assert L.last_launch()[0] == "gemm_frag_kernel" and L.last_launch()[2] > 1
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-5 * np.linalg.norm(ref)
    del graph
    w.close()


def test_three_rows_take_the_same_kernel_whatever_was_called_before():
    """Several k-ranges reduce into rows that the container has from the start: a first call, one in a capture, calls after a larger
    batch and in an explicit workspace run the same launch."""
    N, K, q, g = 264, 8192, 2, 128
    bW, alpha, _ = synth.bcq_layer(N, K, q, g, seed=8)
    x = synth.activations(8, K, seed=9)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    ref = oracle.bcq_matmul_f64(x, bW, alpha.astype(np.float16), None, g)
    w, captured = (L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g) for _ in range(2))
    seen = []

    def three(w, **workspace):
        y = torch.empty((3, N), dtype=torch.float16, device="cuda")
        L.matmul(y, xd, w, 3, **workspace)
        seen.append(L.last_launch())
        return y

    def right(y, rows=3):
        assert np.linalg.norm(y.cpu().numpy() - ref[:rows]) <= 8e-4 * np.linalg.norm(ref[:rows])

    right(three(w))
    assert w.scratch() == (0, 0, 0) and seen[0][0] == "gemm_frag_kernel" and seen[0][2] > 1
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        y = three(captured)
    graph.replay()
    torch.cuda.synchronize()
    right(y)
    for m, dtype, f in ((8, torch.float16, L.matmul), (2, torch.float32, L.matmul_f32)):
        y = torch.empty((m, N), dtype=dtype, device="cuda")
        f(y, xd, w, m)
        right(y, m)
        right(three(w))
    ws = L.Workspace(2 * N, K)
    right(three(w, workspace=ws))
    right(three(w, workspace=ws))
    assert len(set(seen)) == 1, seen
    ws.close()
    del graph
    w.close()
    captured.close()


def _far_apart_in_a_column(N, K, q, g, bias, m):
    """Scales whose exponents differ from group to group of one column from one end of fp16 to the other; activations are zero
    wherever some column's scales are large, so that what the outputs consist of are the products with the small ones."""
    rng = np.random.default_rng(N + K + q)
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + K + m, with_bias=bias)
    G = K // g
    large = np.arange(G) % 2 == 0
    e = np.where(large[:, None], 30000.0 / (q + 1), 2.0 ** rng.integers(-22, -15, (G, 1))) * np.ones((G, N))
    # two columns of each eight have no scale of 8192 or more, one neither large nor small ones
    e[:, 5::8] = np.where(large[:, None], 2.0 ** -3, e[:, 5::8])
    e[:, 6::8] = np.where(large[:, None], 2.0 ** 10, e[:, 6::8])
    e[:, 7::8] = 1.0
    draw = lambda shape: np.abs(rng.normal(1.0, 0.3, shape)) + 0.01
    alpha = (draw((G, q, N)) * e[:, None, :])
    alpha[large, 0, ::8] = 40000.0
    alpha = alpha.astype(np.float16).astype(np.float32)
    if bias:
        q_bias = (draw((G, N)) * e * np.where(rng.random((G, N)) < 0.5, -1, 1)).astype(np.float16).astype(np.float32)
    x = synth.activations(m, K, seed=m)
    x.reshape(m, G, g)[:, large, :] = 0
    return bW, alpha, q_bias, x


@pytest.mark.parametrize("N,K,q,g,bias,m", [
    (264, 1024, 4, 64, True, 64), (264, 1024, 2, 64, False, 130), (136, 2048, 1, 128, False, 200), (128, 512, 1, 32, True, 257),
    (1032, 4096, 3, 256, True, 129)])
def test_split_operand_kernel_scales_far_apart_within_a_column(N, K, q, g, bias, m):
    bW, alpha, q_bias, x = _far_apart_in_a_column(N, K, q, g, bias, m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y = torch.empty((m, N), dtype=torch.float32, device="cuda")
    L.matmul_f32(y, xd, w, m)
    assert L.last_launch()[0] == "gemm_hl_kernel"
    a16, b16 = alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16)
    ref = oracle.bcq_matmul_f64(x, bW, a16, b16, g)
    mag = np.abs(a16.astype(np.float64)).sum(1) + (0 if b16 is None else np.abs(b16.astype(np.float64)))
    size = np.abs(x.astype(np.float64)).reshape(m, K // g, g).sum(2) @ mag
    # fp32 sums as in _run, with weights (2^-22) instead of products with offsets
    bound = ((2 * K / 16 + 64) * 2.0 ** -23 + 2.0 ** -22) * size + 1e-30
    err = np.abs(y.cpu().numpy().astype(np.float64) - ref)
    assert (err <= bound).all(), (err / bound).max()
    # the same per column in the 2-norm, where partial sums of terms of either sign are no larger than the whole (1.5: the
    # spread over 64 rows or more)
    assert (np.linalg.norm(err, axis=0) <= 1.5 * ((2 * K / 16 + 64) * 2.0 ** -23 + 2.0 ** -22) * np.linalg.norm(ref, axis=0)).all()
    w.close()


def _not_finite(N, K, q, g, bias, m, kernel):
    """Rows with an infinite activation give what the planes give, +-alpha_b * x summed: an infinity where all planes of
    that weight agree in sign, else NaN; NaN rows are NaN, and the other rows do not notice."""
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, g, seed=N + K + m, with_bias=bias)
    alpha = np.maximum(alpha, 2.0 ** -10)                 # 0 * inf would be NaN in every column
    x = synth.activations(m, K, seed=m)
    clean = x.copy()
    x[0, K // 3] = np.inf
    x[2, K - 1] = -np.inf
    x[m - 1, 0], x[m - 1, K // 2] = np.inf, -np.inf
    x[1, K // 2] = np.nan
    touched = [0, 1, 2, m - 1]
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // g, q_bias).reserve_batch(m)
    xd = torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)
    y = torch.empty((m, N), dtype=torch.float32, device="cuda")
    a16, b16 = alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16)
    ref = oracle.bcq_matmul_f64(clean, bW, a16, b16, g)
    ref[1] = np.nan
    bits = np.unpackbits(bW.view(np.uint8).reshape(K // 32, q, N, 4), axis=-1, bitorder="little")       # [K / 32, q, N, 32]
    for r in (0, 2, m - 1):
        terms = []
        for k in np.flatnonzero(np.isinf(x[r])):
            planes = np.where(bits[k // 32, :, :, k % 32] == 1, 1.0, -1.0) * a16[k // g].astype(np.float64)
            if b16 is not None:
                planes = np.concatenate([planes, b16[k // g].astype(np.float64)[None]])
            terms.append(planes * np.float64(x[r, k]))
        with np.errstate(invalid="ignore"):
            ref[r] = np.concatenate(terms).sum(0)
    for _ in range(2):
        L.matmul_f32(y, xd, w, m)
        assert L.last_launch()[0] == kernel
        got = y.cpu().numpy()
        for r in touched:
            assert np.array_equal(got[r], ref[r].astype(np.float32), equal_nan=True), r
        rest = [r for r in range(m) if r not in touched]
        assert np.linalg.norm(got[rest] - ref[rest]) <= 1e-5 * np.linalg.norm(ref[rest])
    w.close()


@pytest.mark.parametrize("N,K,q,g,bias,m", [(264, 1024, 4, 128, True, 40), (136, 2048, 2, 64, False, 130), (128, 512, 1, 32, True, 257),
                                            (128, 512, 1, 128, False, 144), (1032, 1024, 3, 256, False, 66)])
def test_split_operand_kernel_activations_not_finite(N, K, q, g, bias, m):
    _not_finite(N, K, q, g, bias, m, "gemm_hl_kernel")


def test_plane_kernel_activations_not_finite():
    _not_finite(264, 1024, 2, 128, False, 20, "gemm_tc_kernel")


@pytest.mark.parametrize("N,K,q,g,bias,m", [(132, 1024, 1, 128, False, 8), (1000, 2048, 3, 64, True, 5), (100, 160, 2, 32, False, 9),
                                            (36, 4128, 3, 96, True, 18), (264, 8192, 2, 512, False, 4)])
def test_register_operand_kernel_activations_not_finite(N, K, q, g, bias, m):
    _not_finite(N, K, q, g, bias, m, "gemm_frag_kernel")


@pytest.mark.parametrize("N,K,q,bias,m", [(1024, 8192, 1, False, 2048), (1024, 8192, 2, False, 2048), (264, 8192, 3, False, 64), (520, 4096, 4, True, 300)])
def test_split_operand_kernel_sums_are_as_close_as_the_plane_kernels(N, K, q, bias, m):
    """Every accumulation of the tensor core cuts its sum off: an fp32 result is no further off than the chains of the plane
    kernel make it, 8 accumulations per plane and 128 k, over 8 k-ranges at these widths."""
    bW, alpha, q_bias = synth.bcq_layer(N, K, q, 128, seed=N + m, with_bias=bias)
    x = synth.activations(m, K, seed=m)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // 128, q_bias).reserve_batch(m)
    y = torch.empty((m, N), dtype=torch.float32, device="cuda")
    L.matmul_f32(y, torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16), w, m)
    assert L.last_launch()[0] == "gemm_hl_kernel"
    rows = np.arange(0, m, max(1, m // 32))
    ref = oracle.bcq_matmul_f64(np.ascontiguousarray(x[rows]), bW, alpha.astype(np.float16), None if q_bias is None else q_bias.astype(np.float16), 128)
    chain = 8 * (q + bias) * (K // 128) / 8
    # 1.8e-8 per accumulation is what the tensor core was measured at; 1.2 for the spread, and the fp32 roundings of the rest
    assert np.linalg.norm(y.cpu().numpy()[rows] - ref) <= (1.2 * 1.8e-8 * chain + 2.0 ** -22) * np.linalg.norm(ref)
    w.close()
