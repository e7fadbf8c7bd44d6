"""The kernels at the sizes and inputs where their paths change, against the
oracle.

* The in-place transforms of the any-size fluid operator: the smallest axes,
  odd rows and slabs (a row pair without its second row), primes above the
  register radices, one to four stages an axis, extra places of the packed
  column on one line (ny = 2), slabs beyond one block. The bound is that of
  the operator's other tests, 1e-5 of max |fp64|; a transform of n values
  rounds each of them about 3 log2(n) times to 6e-8, under 4e-6 for three
  axes of 512.
* The splat's sums: destinations whose candidates come in order, out of
  order, more than fit the list, buckets left unsorted and sorted. Bit-exact.
* The direct kernel's data gradient, with one, two and four planes a tile and
  with and without the ReLU mask: BF16 outputs to 1e-2 of max |ref|, the
  bound of the GEMM path's test (one BF16 rounding is 2^-9), and the GEMM
  path's own bits, its split K included.
* The weight and bias gradients' FP32 sums over K splits and over rows, in
  the order that the kernels state. Bit-exact.
* Interpolation at the volume's borders, at positions just below zero (whose
  fraction is not a float), at integers, and beyond the range of the fast
  floor. Bit-exact.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from atlaswerks_b200 import _lib  # noqa: E402
from atlaswerks_b200 import device as D  # noqa: E402
from atlaswerks_b200.greedy import (DiffOperB200, DiffOperParam, GreedyDeformationDataB200,  # noqa: E402
                                    GreedyIteratorB200, GreedyIteratorParam)
from atlaswerks_b200.ldmm import LDMMIteratorParam  # noqa: E402
from atlaswerks_b200.shooting import LDMMAdShootingIteratorB200, LDMMShootingDefDataB200  # noqa: E402
from atlaswerks_b200.synth import greedy_pair  # noqa: E402
from oracle import identity  # noqa: E402
from oracle import nn_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


@pytest.mark.parametrize("shape", [
    (2, 2, 2), (2, 2, 3), (3, 2, 2), (2, 3, 2), (3, 3, 3), (2, 4, 6),  # [nz, ny, nx]
    (5, 7, 9), (11, 13, 10), (13, 12, 11),
    (17, 18, 16), (16, 17, 34), (19, 16, 23), (7, 62, 31), (109, 4, 6), (6, 109, 38), (8, 6, 181),
    (289, 3, 4), (3, 4, 289),                                          # two primes above the radices
    (96, 20, 24), (20, 243, 12), (250, 6, 10), (512, 6, 4), (4, 512, 6), (4, 6, 509),
    (3, 330, 257), (4, 299, 300)])
@pytest.mark.parametrize("inverse", [True, False])
def test_fluid_operator_any_axis(oracle, shape, inverse):
    rng = np.random.default_rng(31)
    sp = (1.0, 1.3, 0.8)
    f = rng.normal(0, 1, (3,) + shape).astype(np.float32)
    want = oracle.fluid_f64(f, sp, inverse=inverse)
    op = DiffOperB200()
    op.SetSize(shape[::-1], sp, DiffOperParam())
    v = cu(f)
    (op.ApplyInverseOperator if inverse else op.ApplyOperator)(v)
    err = np.abs(host(v).astype(np.float64) - want).max() / np.abs(want).max()
    assert err <= 1e-5, err
    assert not op.TimedOut()


@pytest.mark.parametrize("shape,pairs", [
    ((120, 45, 181), 0), ((120, 154, 155), 0), ((220, 167, 98), 0), ((120, 145, 153), 0), ((280, 81, 205), 0),
    ((3, 245, 257), 16), ((5, 241, 271), 22), ((3, 331, 259), 0)])
@pytest.mark.parametrize("inverse", [True, False])
def test_fluid_prime_stage_leaves_one_over(oracle, shape, pairs, inverse):
    """A prime above the register radices over an odd number of butterflies, the last of which falls into a group
    of threads of its own: 385 in groups of 96, 49 in 12, 205 in 51, 23 in 11; on split grids the last batch's 11
    or 11 lines of `pairs`."""
    rng = np.random.default_rng(41)
    sp = (1.0, 1.3, 0.8)
    f = rng.normal(0, 1, (3,) + shape).astype(np.float32)
    want = oracle.fluid_f64(f, sp, inverse=inverse)
    op = DiffOperB200()
    op.SetSize(shape[::-1], sp, DiffOperParam())
    if pairs:
        _lib.check(_lib.lib().aw_fluid_set_shapes(op._h, pairs, 16, 8))
    v = cu(f)
    (op.ApplyInverseOperator if inverse else op.ApplyOperator)(v)
    err = np.abs(host(v).astype(np.float64) - want).max() / np.abs(want).max()
    assert err <= 1e-5, err
    assert not op.TimedOut()


# Slabs that fit one block without room for two more buffers of a batch, the largest that do (120 x 470 and
# 312 x 182 would but for the block's barrier), and larger ones.
@pytest.mark.parametrize("shape", [(3, 224, 224), (2, 220, 240), (3, 240, 208), (2, 200, 256), (2, 100, 512),
                                   (2, 470, 120), (3, 182, 312), (2, 469, 119), (2, 472, 120), (2, 184, 312)])
@pytest.mark.parametrize("inverse", [True, False])
def test_fluid_slabs_at_the_limit_of_one_block(oracle, shape, inverse):
    rng = np.random.default_rng(42)
    sp = (1.0, 1.3, 0.8)
    f = rng.normal(0, 1, (3,) + shape).astype(np.float32)
    want = oracle.fluid_f64(f, sp, inverse=inverse)
    op = DiffOperB200()
    op.SetSize(shape[::-1], sp, DiffOperParam())
    v = cu(f)
    (op.ApplyInverseOperator if inverse else op.ApplyOperator)(v)
    err = np.abs(host(v).astype(np.float64) - want).max() / np.abs(want).max()
    assert err <= 1e-5, err
    assert not op.TimedOut()


@pytest.mark.parametrize("nz,fits", [(152, 1), (293, 1), (294, 0), (512, 0)])
def test_fluid_z_tile_of_32_columns(oracle, nz, fits):
    """Taken wherever its shared memory is there; a refused shape leaves the plan as it was."""
    rng = np.random.default_rng(43)
    f = rng.normal(0, 1, (3, nz, 5, 36)).astype(np.float32)
    op = DiffOperB200()
    op.SetSize((36, 5, nz), (1.0, 1.0, 1.0), DiffOperParam())
    L = _lib.lib()
    _lib.check(L.aw_fluid_set_shapes(op._h, 1, 1, 8))
    want = host(op.ApplyInverseOperator(cu(f))).copy()
    assert (L.aw_fluid_set_shapes(op._h, 1, 1, 32) == 0) == bool(fits)
    assert np.array_equal(host(op.ApplyInverseOperator(cu(f))), want)
    assert L.aw_fluid_set_shapes(op._h, 1, 1, 16) == 0
    assert np.array_equal(host(op.ApplyInverseOperator(cu(f))), want)


@pytest.mark.parametrize("shape", [(12, 11, 10), (7, 18, 30), (16, 32, 16)])
@pytest.mark.parametrize("k", [70, -70])
def test_fluid_parameters_scale(shape, k):
    """alpha, beta and gamma times a power of two scale every wavenumber's matrix by it, exactly: so does the
    result, up to diagonal terms whose squares are no floats."""
    rng = np.random.default_rng(44)
    f = rng.normal(0, 1, (3,) + shape).astype(np.float32)
    out = []
    for s in (1.0, 2.0 ** k):
        op = DiffOperB200()
        op.SetSize(shape[::-1], (1.0, 1.3, 0.8), DiffOperParam(0.01 * s, 0.01 * s, 0.001 * s))
        out.append((host(op.ApplyInverseOperator(cu(f))).copy(), host(op.ApplyOperator(cu(f))).copy()))
    assert np.isfinite(out[1][0]).all() and np.isfinite(out[1][1]).all()
    assert np.array_equal(out[1][0] * np.float32(2.0 ** k), out[0][0])
    assert np.array_equal(out[1][1] * np.float32(2.0 ** -k), out[0][1])


@pytest.mark.parametrize("shape", [(12, 11, 10), (9, 17, 131), (20, 18, 16)])
@pytest.mark.parametrize("scale", [1.0, 0.85, 0.7, 0.55, 0.42, 0.3])
@pytest.mark.parametrize("jitter", [0.0, 0.3])
def test_splat_candidate_counts(oracle, shape, scale, jitter):
    """scale^-3 sources a cell: 1, 1.6, 2.9, 6, 13, 37; eight times that per destination."""
    rng = np.random.default_rng(32)
    img = rng.normal(0, 1, shape).astype(np.float32)
    h = identity(shape) * np.float32(scale) + rng.normal(0, 1, (3,) + shape) * jitter + 0.3
    h = h.astype(np.float32)
    want = oracle.splat(img, h, 0.25)
    for _ in range(2):  # the arrival order inside a bucket may differ
        assert np.array_equal(host(D.splat(cu(img), cu(h), 0.25)), want)


@pytest.mark.parametrize("shape", [(1, 2, 340), (160, 160, 160), (160, 161, 160)])
def test_splat_scan_sizes(oracle, shape):
    """Cells of two blocks of the scan, and just below and above the most
    whose sums its last kernel adds up itself (4096 blocks of 1024)."""
    rng = np.random.default_rng(37)
    img = rng.normal(0, 1, shape).astype(np.float32)
    h = (identity(shape) + rng.normal(0, 0.4, (3,) + shape)).astype(np.float32)
    assert np.array_equal(host(D.splat(cu(img), cu(h), 0.0)), oracle.splat(img, h, 0.0))


@pytest.mark.parametrize("shape", [(12, 11, 10), (16, 32, 16)])
def test_a_failed_launch_is_reported_once(shape):
    """An operator called on a stream whose capture was given up reports that; a call on another stream does not."""
    import ctypes
    op = DiffOperB200()
    op.SetSize(shape[::-1], (1.0, 1.0, 1.0), DiffOperParam())
    v = torch.zeros((3,) + shape, device="cuda")
    img, g = torch.rand(shape, device="cuda"), torch.zeros((3,) + shape, device="cuda")
    L, rt = _lib.lib(), ctypes.CDLL("libcudart.so.12")
    s = torch.cuda.Stream()
    st = ctypes.c_void_p(s.cuda_stream)
    torch.cuda.synchronize()
    nz, ny, nx = shape
    assert rt.cudaStreamBeginCapture(st, 2) == 0  # relaxed: other streams go on
    try:
        assert rt.cudaStreamSynchronize(st) != 0  # not allowed in a capture, which ends it
        rt.cudaGetLastError()
        assert L.aw_fluid_apply(op._h, *[t.data_ptr() for t in v], 1, st) != 0
        rc = L.aw_gradient(img.data_ptr(), *[t.data_ptr() for t in g], nx, ny, nz, 1.0, 1.0, 1.0, 0, None)
        msg = L.aw_last_error()
    finally:
        graph = ctypes.c_void_p()
        rt.cudaStreamEndCapture(st, ctypes.byref(graph))
        rt.cudaGetLastError()
    assert rc == 0, msg
    assert np.isfinite(host(op.ApplyInverseOperator(v))).all()


def test_adjoint_shooting_memory():
    """The T + 1 kept sorts share one buffer of products: a handle at 80 x 96 x 112 with T = 5 stays below the
    fields' and the sorts' own memory plus one such buffer, which T + 2 of them would exceed by 90 MB."""
    nz, ny, nx, T = 80, 96, 112, 5
    n, cells = nz * ny * nx, (nz + 1) * (ny + 1) * (nx + 1)
    z = torch.zeros((nz, ny, nx), device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    it = LDMMAdShootingIteratorB200((nx, ny, nz), n_time_steps=T)
    it.SetScaleLevel((nx, ny, nz), (1.0, 1.0, 1.0), LDMMIteratorParam(DiffOperParam(), 1.0, 0.01, False))
    data = LDMMShootingDefDataB200(z, z, (1.0, 1.0, 1.0))
    it.Iterate(data)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    floats = (T + 11 + 3 * 2) * n + (3 * T + 6 * (T + 1) + T + 6) * n  # the handle's fields, the iteration's, the data's
    sorts = (T + 2) * (2 * cells + n)
    assert used <= 4 * (floats + sorts + 8 * n) + (64 << 20), used / 2 ** 20


@pytest.mark.parametrize("grid", [(1, 8, 32, 16), (2, 6, 32, 24), (1, 3, 32, 16), (1, 32, 64, 64)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 16), (16, 32), (32, 32)])
@pytest.mark.parametrize("masked", [True, False])
def test_conv_dgrad_direct(grid, cin, cout, masked):
    B, DD, H, W = grid
    rng = np.random.default_rng(36)
    dy = O.bf16(rng.normal(0, 1, grid + (cout,)).astype(np.float32))
    w = O.bf16(rng.normal(0, 0.1, (cout, 27, cin)).astype(np.float32))
    mask = O.bf16(rng.normal(0, 1, grid + (cin,)).astype(np.float32)) if masked else None
    want = O.conv_dgrad(dy, w, mask if masked else np.ones(grid + (cin,), np.float32))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).cuda()  # noqa: E731
    dyd, wtd, md = dev(dy), dev(w.transpose(2, 1, 0)), dev(mask) if masked else None
    dx = torch.zeros((B * DD * H * W, cin), dtype=torch.bfloat16, device="cuda")
    rc = _lib.lib().aw_nn_conv3d_dgrad(dyd.data_ptr(), B, DD, H, W, cout, wtd.data_ptr(), cin, 27,
                                       md.data_ptr() if masked else None, dx.data_ptr(), None, 0, None)
    assert rc == 0, _lib.lib().aw_last_error()
    got = host(dx.float()).reshape(want.shape)
    assert np.abs(got - want).max() <= 1e-2 * np.abs(want).max()


@pytest.mark.parametrize("grid", [(1, 32, 32, 32), (1, 28, 32, 24), (1, 40, 48, 32), (2, 8, 32, 40)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 16), (16, 32), (32, 32)])
@pytest.mark.parametrize("scratch", [True, False])
def test_conv_dgrad_bits_do_not_depend_on_the_path(grid, cin, cout, scratch):
    """With the scratch of aw_nn_conv3d_scratch_floats the GEMM splits K on the small grids (32^3: in three)
    and not on the others; without it, nowhere."""
    B, DD, H, W = grid
    rng = np.random.default_rng(38)
    dev = lambda a: torch.from_numpy(a).to(torch.bfloat16).cuda()  # noqa: E731
    dy = dev(rng.normal(0, 1, grid + (cout,)).astype(np.float32))
    wt = dev(rng.normal(0, 0.1, (cin, 27, cout)).astype(np.float32))
    mask = dev(rng.normal(0, 1, grid + (cin,)).astype(np.float32))
    L = _lib.lib()
    n = int(L.aw_nn_conv3d_scratch_floats(*grid, cin, cout, 27)) if scratch else 0
    sc = torch.zeros(max(n, 1), device="cuda")
    got = []
    for gemm in (0, 1):
        dx = torch.zeros((B * DD * H * W, cin), dtype=torch.bfloat16, device="cuda")
        L.aw_nn_set_gemm_only(gemm)
        try:
            rc = L.aw_nn_conv3d_dgrad(dy.data_ptr(), B, DD, H, W, cout, wt.data_ptr(), cin, 27, mask.data_ptr(),
                                      dx.data_ptr(), sc.data_ptr() if n else None, n, None)
        finally:
            L.aw_nn_set_gemm_only(0)
        assert rc == 0, L.aw_last_error()
        got.append(dx)
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("grid", [(1, 31, 32, 33), (1, 29, 36, 32), (1, 5, 7, 9)])  # 32736, 33408 and 315 rows
@pytest.mark.parametrize("cin,cout,taps", [(48, 16, 27), (96, 32, 27), (32, 16, 27), (64, 64, 1), (48, 48, 1)])
def test_conv_operand_loaders(grid, cin, cout, taps):
    """Below 64 columns the GEMM's rows come 64 bytes of eight rows a warp from 48 channels and 32768 rows on, else
    a row a thread: ragged last tiles on either side, to the bound of the GEMM's other tests."""
    B, DD, H, W = grid
    rng = np.random.default_rng(45)
    x = O.bf16(rng.normal(0, 1, grid + (cin,)).astype(np.float32))
    w = O.bf16(rng.normal(0, 0.1, (cout, taps, cin)).astype(np.float32))
    b = rng.normal(0, 0.1, cout).astype(np.float32)
    want = O.conv_fwd(x, w, b, relu=False)
    xd, wd = (torch.from_numpy(a).to(torch.bfloat16).cuda() for a in (x, w))
    bd = torch.from_numpy(b).cuda()
    out = torch.zeros((B * DD * H * W, cout), device="cuda")
    rc = _lib.lib().aw_nn_conv3d_fwd(xd.data_ptr(), B, DD, H, W, cin, wd.data_ptr(), bd.data_ptr(), cout, taps, 0,
                                     None, out.data_ptr(), None, 0, None)
    assert rc == 0, _lib.lib().aw_last_error()
    assert np.abs(host(out).reshape(want.shape) - want).max() <= 1e-3 * np.abs(want).max()


@pytest.mark.parametrize("grid,splits", [((1, 8, 8, 8), 1), ((1, 8, 8, 8), 3), ((2, 8, 16, 64), 130),
                                         ((1, 8, 48, 48), 288)])
@pytest.mark.parametrize("cin,cout,taps", [(16, 16, 1), (32, 16, 27), (16, 48, 27)])
def test_wgrad_splits_in_order(grid, splits, cin, cout, taps):
    """dW is the sum of the splits' partial results, which the call leaves in its scratch, first to last."""
    rng = np.random.default_rng(39)
    B, DD, H, W = grid
    x = torch.from_numpy(rng.normal(0, 1, grid + (cin,)).astype(np.float32)).to(torch.bfloat16).cuda()
    dy = torch.from_numpy(rng.normal(0, 1, grid + (cout,)).astype(np.float32)).to(torch.bfloat16).cuda()
    L = _lib.lib()
    part = torch.zeros(int(L.aw_nn_wgrad_scratch_floats(cin, cout, taps, splits)), device="cuda")
    dw = torch.zeros((cout, taps, cin), device="cuda")
    rc = L.aw_nn_conv3d_wgrad(x.data_ptr(), dy.data_ptr(), B, DD, H, W, cin, cout, taps, splits, part.data_ptr(),
                              dw.data_ptr(), None)
    assert rc == 0, L.aw_last_error()
    used = -(-B * DD * H * W // (-(-(-(-B * DD * H * W // splits)) // 64) * 64))  # splits of whole 64-voxel steps
    want = np.zeros(dw.shape, np.float32)
    for p in host(part).reshape(splits, cout, taps, cin)[:used]:
        want = want + p
    assert np.array_equal(host(dw), want)


@pytest.mark.parametrize("cout", [1, 7, 16, 24, 32, 64, 128, 192, 256])
@pytest.mark.parametrize("rows", [1, 511, 512, 1234, 512 * 130 + 3])
def test_bias_sums_in_order(rows, cout):
    """Blocks of 512 rows: every (256 / cout)-th row from each of the first ones, these sums first to last, then
    the blocks first to last."""
    rng = np.random.default_rng(40)
    dy = torch.from_numpy(rng.normal(0, 1, (rows, cout)).astype(np.float32)).to(torch.bfloat16)
    L = _lib.lib()
    sc = torch.zeros(int(L.aw_nn_bias_scratch_floats(rows, cout)), device="cuda")
    db = torch.zeros(cout, device="cuda")
    d = dy.cuda()
    assert L.aw_nn_bias_grad(d.data_ptr(), rows, cout, sc.data_ptr(), db.data_ptr(), None) == 0
    blocks, groups = -(-rows // 512), 256 // cout
    steps = -(-512 // groups)
    y = np.zeros((blocks, 512, cout), np.float32)
    y.reshape(-1, cout)[:rows] = dy.float().numpy()
    y = np.concatenate([y, np.zeros((blocks, steps * groups - 512, cout), np.float32)], 1)
    y = y.reshape(blocks, steps, groups, cout)  # adding a zero keeps a sum's bits

    def in_order(a, axis):
        t = np.zeros(np.delete(a.shape, axis), np.float32)
        for k in range(a.shape[axis]):
            t = t + np.take(a, k, axis)
        return t
    want = in_order(in_order(in_order(y, 1), 1), 0)
    assert np.array_equal(host(db), want)


@pytest.mark.parametrize("shape,sp,max_pert", [((64, 64, 64), (1.0, 1.0, 1.0), 0.5),
                                               ((128, 128, 128), (1.0, 1.0, 1.0), 0.5),
                                               ((16, 32, 128), (2.0, 1.3, 0.8), 3.0),   # 65536: fused
                                               ((32, 32, 128), (1.0, 1.3, 0.8), 0.5),   # the next: separate
                                               ((32, 64, 32), (1.0, 1.0, 1.0), 2.0),    # 65536, narrow: fused
                                               ((32, 32, 32), (1.0, 1.0, 1.0), 0.5),    # below: separate
                                               ((16, 64, 256), (1.0, 1.0, 1.5), 3.0)])
def test_fused_update_on_either_side_of_its_rule(shape, sp, max_pert):
    """One kernel for the inverse transform and the update (2), two (0) and the rule's choice (1): the same bits,
    with the float interpolation too where both run it."""
    I0, I1 = greedy_pair(shape, seed=13)
    L = _lib.lib()

    def run(fused, fast):
        it = GreedyIteratorB200(shape[::-1], spacing=sp)
        it.SetScaleLevel(shape[::-1], sp, GreedyIteratorParam(DiffOperParam(0.01, 0.01, 0.001), max_pert))
        _lib.check(L.aw_greedy_set_fused_update(it._h, fused))
        it.SetFastInterpolation(fast)
        d = GreedyDeformationDataB200(cu(I0), cu(I1), spacing=sp)
        it.Run(d, 5, update_first=True)
        return host(d.Def1To0()).copy(), it.Energies()
    h, e = run(0, False)
    assert np.abs(h - identity(shape)).max() > 0.1
    for fused in (1, 2):
        got = run(fused, False)
        assert np.array_equal(got[0], h) and np.array_equal(got[1], e)
    f1, f2 = run(1, True), run(2, True)
    assert np.array_equal(f1[0], f2[0]) and np.array_equal(f1[1], f2[1])
    assert not np.array_equal(f1[0], h)  # the float tree ran


@pytest.mark.parametrize("shape", [(32, 32, 64), (24, 20, 28), (6, 260, 250)])
@pytest.mark.parametrize("reps", [1, 2, 25])
def test_profile_leaves_one_iteration(shape, reps):
    """The stages run on an iteration's own data however often each is repeated: h_out is the iteration's result,
    bit for bit, on split slabs too."""
    import ctypes
    I0, I1 = (cu(a) for a in greedy_pair(shape, seed=13))
    it = GreedyIteratorB200(shape[::-1])
    it.SetScaleLevel(shape[::-1], (1.0, 1.0, 1.0), GreedyIteratorParam(DiffOperParam(), 0.5))
    d = GreedyDeformationDataB200(I0, I1)
    it.UpdateStepSizeNextIteration()
    it.Iterate(d)
    want = host(d.Def1To0()).copy()
    h, ho = cu(identity(shape)), torch.zeros((3,) + shape, device="cuda")
    ms, z = (ctypes.c_float * 8)(), [None] * 3
    _lib.check(_lib.lib().aw_greedy_profile(it._h, I0.data_ptr(), I1.data_ptr(), *[t.data_ptr() for t in h],
                                            *[t.data_ptr() for t in ho], *z, *z, reps, None, ms))
    assert np.abs(want - identity(shape)).max() > 0.2
    assert np.array_equal(host(ho), want)


def _edge_field(shape, rng):
    """Positions all over the borders, a tenth of them special."""
    h = identity(shape) + rng.normal(0, 0.6, (3,) + shape).astype(np.float32)
    special = np.float32([0.0, -0.0, -1e-10, -1e-30, 1e-10, -0.5, 0.5, 1.0, -1.0, 2.0 ** 21, -2.0 ** 21,
                          2.0 ** 22 + 1, 2.0 ** 23 - 1, -2.0 ** 23 - 1, 1e9])
    pick = rng.random(h.shape) < 0.1
    h[pick] = special[rng.integers(0, special.size, int(pick.sum()))]
    for a in range(3):  # the far border too
        n = shape[2 - a]
        far = rng.random(h[a].shape) < 0.05
        h[a][far] = (n - 1) + rng.choice(np.float32([0.0, -1e-6, 1e-6, 0.5, 1.0]), int(far.sum()))
    return h.astype(np.float32)


@pytest.mark.parametrize("shape", [(8, 9, 33), (5, 4, 130), (2, 2, 2)])
def test_apply_at_the_edges(oracle, shape):
    rng = np.random.default_rng(33)
    img = rng.random(shape, dtype=np.float32)
    h = _edge_field(shape, rng)
    assert np.array_equal(host(D.apply(cu(img), cu(h), 0.7)), oracle.apply(img, h, 0.7))


@pytest.mark.parametrize("shape", [(8, 9, 33), (2, 2, 2)])
@pytest.mark.parametrize("bg", range(4))
@pytest.mark.parametrize("sp", [(1.0, 1.0, 1.0), (1.5, 0.75, 1.2)])
def test_compose_at_the_edges(oracle, shape, bg, sp):
    rng = np.random.default_rng(34)
    g = identity(shape) + rng.normal(0, 1, (3,) + shape).astype(np.float32)
    v = rng.normal(0, 1, (3,) + shape).astype(np.float32)
    h = _edge_field(shape, rng)
    got = host(D.compose_vh(cu(v), cu(h), sp, 1.0, -1, bg))
    assert np.array_equal(got, oracle.compose_vh(v, h, sp, -1, bg))
    u = ((h - identity(shape)) * np.float32(sp).reshape(3, 1, 1, 1)).astype(np.float32)
    got = host(D.compose_hv(cu(g), cu(u), sp, 1.0, 1, bg))
    assert np.array_equal(got, oracle.compose_hv(g, u, sp, 1, bg))


@pytest.mark.parametrize("sp", [(1.0, 1.2, 1.0), (1.5, 0.75, 1.25), (1.2, 0.9, 2.06452), (2.0, 0.5, 1.0)])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 129), (6, 2, 40)])
@pytest.mark.parametrize("wrap", [False, True])
def test_gradient_kernels_at_the_borders(oracle, sp, shape, wrap):
    """Float and other spacings, one-sided and wrapped differences, axes of two voxels. Bit-exact."""
    rng = np.random.default_rng(46)
    img = rng.normal(0, 1, shape).astype(np.float32)
    assert np.array_equal(host(D.gradient(cu(img), sp, wrap)), oracle.gradient(img, sp, wrap))


@pytest.mark.parametrize("sp", [(1.5, 0.75, 1.25), (1.2, 0.9, 2.06452), (2.0, 0.5, 1.0)])
def test_gradient_divisors(oracle, sp):
    """Spacings divided in float (exactly floats), in double, and multiplied."""
    rng = np.random.default_rng(35)
    img = rng.normal(0, 1, (7, 9, 12)).astype(np.float32)
    assert np.array_equal(host(D.gradient(cu(img), sp)), oracle.gradient(img, sp, False))
