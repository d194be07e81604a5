"""Kernels at the sizes where their tiles, chunks and remainders meet, against the oracle or the reference."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import oracle as O  # noqa: E402
import robtop_b200 as rb  # noqa: E402
from gpu_common import E, NU, P, rel_err  # noqa: E402


def _perforated(nx, ny, nz, seed, sup, skip=1):
    """A box with voids and scattered supports, and its oracle hierarchy."""
    r = np.random.default_rng(seed)
    eact = (r.random((nz, ny, nx)) < 0.85).astype(np.uint8)
    rho = ((0.1 + 0.9 * r.random(eact.shape)) * eact).astype(np.float32)
    vfix = np.zeros((nz + 1, ny + 1, nx + 1), np.uint8)
    if sup:
        vfix[0] = 1
        vfix[r.random(vfix.shape) < 0.03] = 1
    ctx = rb.Context(0)
    G = rb.HierarchyGrid(ctx, rb.default_params(mode=rb.MODE_WSFF if sup else rb.MODE_NSFF, youngs_modulus=E,
                                                poisson_ratio=NU, power_penalty=P, skip_layer1=skip))
    G.genFromBox(eact)
    G[0].setRho(rho.ravel())
    G.set_support(vfix)
    H = O.Hierarchy(eact, rho, vfix if sup else None, p=P, E=E, nu=NU, no_support=not sup,
                    skip=bool(skip))
    G.update_stencil()
    H.set_weights(G[0].getPenalty())  # the device's FP32 powf weights
    H.update_stencil()
    return ctx, G, H, r


# node columns finished per warp 30, node rows per block 7 (FP32, and FP64 smoothing), 11 (FP64): boxes one below,
# at and above these, and z-chunks that end inside the box, at its end and beyond it
@pytest.mark.parametrize("nx,ny,nz,zc", [(29, 6, 9, 1), (30, 7, 16, 2), (31, 13, 8, 3), (59, 10, 7, 64), (60, 11, 15, 16),
                                         (12, 21, 17, 5), (95, 8, 8, 4)])
@pytest.mark.parametrize("sup", [True, False])
def test_face_march_edges(nx, ny, nz, zc, sup):
    ctx, G, H, r = _perforated(nx, ny, nz, nx + ny, sup)
    L = rb.lib()
    for prec in (rb.FP64, rb.FP32):
        for m in range(4):
            rb._capi.check(L.rt_set_tuning(G.handle, prec, m, 8, 1, zc), ctx.handle)
    act = np.tile(G[0].getVact(), 3).astype(bool)
    u = r.standard_normal(3 * G[0].nv)
    u[~act] = np.nan  # values of nodes without elements are not read into any result
    f = r.standard_normal(3 * G[0].nv) * act
    uo = np.where(act, u, 0.0)
    G[0].setDisplacement(u)
    G[0].setForce(f)
    G[0].update_residual()
    want = [np.zeros_like(u) for _ in range(4)]
    O.lib().or_fine_residual(H.lv(0), O.ptr(H.KE), O.ptr(uo), O.ptr(f), O.ptr(want[0]))
    want[1] = H.applyK(uo)
    ujac, tmp = uo.copy(), np.zeros_like(u)
    O.lib().or_fine_jacobi(H.lv(0), O.ptr(H.KE), O.ptr(ujac), O.ptr(f), 0.6, O.ptr(tmp))
    H.set_lmax([G.smoother_lmax(i) for i in range(H.nlev - 1)])
    d = np.zeros_like(u)
    O.lib().or_fine_cheby(H.lv(0), O.ptr(H.KE), O.ptr(uo), O.ptr(f), O.ptr(want[3]), O.ptr(d), 0)
    # FP64: the sums of 8 elements in another order; FP32: the tolerance of the other FP32 kernels' tests
    assert rel_err(G[0].getResidual(), want[0]) < 1e-11
    assert rel_err(G[0].applyK(u), want[1]) < 1e-11
    for smoother, w in ((rb.SMOOTH_JACOBI, ujac), (rb.SMOOTH_CHEBY, want[3])):
        G[0].setDisplacement(u)
        G[0].smooth(smoother, 1, 0.6)
        assert rel_err(G[0].getDisplacement(), w) < 1e-10
    G[0].setDisplacement(u)
    for m, w in ((0, want[0]), (1, want[1]), (2, ujac), (3, want[3])):
        rb._capi.check(L.rt_fine_kernel_f32(G.handle, m, 0.6), ctx.handle)
        assert rel_err(G[0].getResidual(), w) < 2e-6
    G.close()
    ctx.close()


# the dot products that come with the march (u . K u in both precisions) and with the step from zero (f . D^-1 f), at the
# same remainders: the smoother bound is 30 of each, and two CG iterations are no further apart than their alpha and beta
@pytest.mark.parametrize("nx,ny,nz,zc", [(29, 6, 9, 1), (30, 7, 16, 2), (31, 13, 8, 3), (59, 10, 7, 64), (60, 11, 15, 16),
                                         (12, 21, 17, 5), (95, 8, 8, 4)])
@pytest.mark.parametrize("sup", [True, False])
def test_face_march_dots(nx, ny, nz, zc, sup):
    ctx, G, H, r = _perforated(nx, ny, nz, nx + ny, sup)
    G.set_tiles(8, 1, zc)
    G.update_stencil()
    # the largest Ritz value of the same 30 steps in another order of summation
    assert abs(G.smoother_lmax(0) - H.LA[0].lmax) <= 1e-6 * H.LA[0].lmax
    if sup:  # without supports the solves project, which the oracle's do not
        b = r.standard_normal(3 * G[0].nv) * np.tile(G[0].getVact(), 3) * (1 - np.tile(H.arrs[0]["vfix"], 3))
        p = G.params
        p.pre_sweeps = p.post_sweeps = 2
        p.jacobi_omega = 0.5
        # FP64: rounding, amplified by the 1e3 contrast; FP32 cycles and vectors: as in test_tail_cycle_edges
        for prec, krylov, smoother, so, tol in ((rb.FP64, 0, rb.SMOOTH_JACOBI, O.SMOOTH_JACOBI, 1e-9),
                                                (rb.FP32, 1, rb.SMOOTH_CHEBY, O.SMOOTH_CHEBY, 1e-3)):
            p.precision, p.krylov_fp32, p.smoother = prec, krylov, smoother
            G.set_params(p)
            G.update_stencil()
            G[0].setForce(b)
            G[0].reset_displacement()
            G.pcg(1e-14, 2)
            want, its, _ = H.pcg(b, tol=1e-14, maxit=2, smoother=so, npre=2, npost=2, omega=0.5)
            assert its == 2 and rel_err(G[0].getDisplacement(), want) < tol
    G.close()
    ctx.close()


# the weight-gradient patches are 8 x 16 voxels by 1 plane, or 2 on the last box: remainders in each axis, one voxel past a patch,
# and the smallest boxes the network takes
@pytest.mark.parametrize("dims", [(9, 17, 8), (8, 16, 8), (33, 15, 12), (25, 8, 9), (34, 17, 25)])
def test_unet_weight_gradient_edges(dims):
    import unet_ref
    from robtop_b200 import learned

    ctx = rb.Context(0)
    net = learned.UNet(ctx, *dims, seed=9)
    p = net.get_params()
    g = torch.Generator().manual_seed(sum(dims))
    V = dims[0] * dims[1] * dims[2]
    inp = torch.randn(V, 16, generator=g).to(torch.bfloat16)
    tgt = torch.randn(V, 3, generator=g)
    _, want, _ = unet_ref.loss_and_grads(p, inp.float(), tgt, dims, emulate_bf16=True)
    _, got = net.gradients(inp.cuda(), tgt.cuda())
    # the bounds of test_unet_gradients_match_reference: bf16 rounding of every layer's gradient and flipped ReLU
    # masks; a wrong tap, transpose or missing patch gives a cosine far from 1
    cos = float(got @ want) / (np.linalg.norm(got) * np.linalg.norm(want))
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 5e-2 and cos > 0.999
    net.close()
    ctx.close()


def _hier(nx, ny, nz, seed, sup=True, skip=1, **kw):
    """A box with random densities and a clamped face, no oracle level beyond the occupancy."""
    r = np.random.default_rng(seed)
    eact = np.ones((nz, ny, nx), np.uint8)
    rho = (0.1 + 0.9 * r.random(eact.shape)).astype(np.float32)
    vfix = np.zeros((nz + 1, ny + 1, nx + 1), np.uint8)
    if sup:
        vfix[:, :, 0] = 1
    ctx = rb.Context(0)
    G = rb.HierarchyGrid(ctx, rb.default_params(mode=rb.MODE_WSFF, youngs_modulus=E, poisson_ratio=NU,
                                                power_penalty=P, skip_layer1=skip, **kw))
    G.genFromBox(eact)
    G[0].setRho(rho.ravel())
    G.set_support(vfix)
    return ctx, G, eact, rho, vfix, r


# the ratio-4 restriction's block owns 31 coarse columns (124 fine) and 4 rows, and several coarse planes per block
# once the blocks fill the GPU (the last box); the prolongation marches several cells there
@pytest.mark.parametrize("dims", [(123, 9, 9), (125, 17, 5), (249, 13, 30), (250, 180, 130)])
def test_transfer_edges(dims):
    ctx, G, eact, rho, vfix, r = _hier(*dims, seed=dims[0], sup=False)
    H = O.Hierarchy(eact, rho, None, p=P, E=E, nu=NU, no_support=True)
    rf = r.standard_normal(3 * G[0].nv)
    G[0].setResidual(rf)
    G[1].restrict_residual()
    fc = np.zeros(3 * G[1].nv)
    O.lib().or_restrict(H.lv(0), H.lv(1), O.ptr(rf), O.ptr(fc))
    assert rel_err(G[1].getForce(), fc) < 1e-13
    uc, uf = r.standard_normal(3 * G[1].nv), r.standard_normal(3 * G[0].nv)
    G[1].setDisplacement(uc)
    G[0].setDisplacement(uf)
    G[0].prolongate_correction()
    O.lib().or_prolong_add(H.lv(0), H.lv(1), O.ptr(uc), O.ptr(uf))
    assert rel_err(G[0].getDisplacement(), uf) < 1e-13
    G.close()
    ctx.close()


# finest Gauss-Seidel: 8 nodes of a colour per warp, 32 per block; colours with odd and even row lengths, nodes on every
# face with and without an element on either side, NaN in nodes that no element holds
@pytest.mark.parametrize("nx,ny,nz", [(15, 7, 8), (16, 8, 7), (17, 9, 9), (40, 7, 7)])
@pytest.mark.parametrize("sup", [True, False])
def test_fine_gauss_seidel_edges(nx, ny, nz, sup):
    ctx, G, H, r = _perforated(nx, ny, nz, nx + nz, sup)
    act = np.tile(G[0].getVact(), 3).astype(bool)
    u = r.standard_normal(3 * G[0].nv)
    u[~act] = np.nan
    f = r.standard_normal(3 * G[0].nv) * act
    for smoother, back in ((rb.SMOOTH_GS, 0), (rb.SMOOTH_SGS, 1)):
        G[0].setDisplacement(u)
        G[0].setForce(f)
        G[0].smooth(smoother, 1)
        uo = np.where(act, u, 0.0)
        O.lib().or_fine_gs(H.lv(0), O.ptr(H.KE), O.ptr(uo), O.ptr(f), back)
        # 168 terms per row and 8 colours in a chain, each product to 2^-53
        assert rel_err(G[0].getDisplacement()[act], uo[act]) < 1e-10
    G.close()
    ctx.close()


# both lane counts of the stencil levels' Gauss-Seidel: a warp per node, and 4 lanes once a colour has ~19k nodes
@pytest.mark.parametrize("dims", [(20, 12, 10), (130, 98, 98)])
def test_level_gauss_seidel_lane_counts(dims):
    ctx, G, eact, rho, vfix, r = _hier(*dims, seed=3, skip=0)
    H = O.Hierarchy(eact, rho, vfix, p=P, E=E, nu=NU, skip=False)
    G.update_stencil()
    st = G[1].getStencil()
    H.arrs[1]["st"][:] = st
    u, f = r.standard_normal(3 * G[1].nv), r.standard_normal(3 * G[1].nv)
    for smoother, back in ((rb.SMOOTH_GS, 0), (rb.SMOOTH_SGS, 1)):
        G[1].setDisplacement(u)
        G[1].setForce(f)
        G[1].smooth(smoother, 1)
        uo = u.copy()
        O.lib().or_st_gs(H.lv(1), O.ptr(uo), O.ptr(f), back)
        assert rel_err(G[1].getDisplacement(), uo) < 1e-10
    G.close()
    ctx.close()


# the filter's shared-memory tiles (32 x 8 x 8 elements, radius up to 3 elements) and the general kernel past them; the
# OC update's vector loads (element counts with every remainder of 4), the default damping and another
@pytest.mark.parametrize("dims", [(33, 9, 9), (31, 7, 17), (13, 7, 5), (64, 16, 8)])
@pytest.mark.parametrize("radius", [1.0, 1.6, 2.0, 3.2, 4.5])
def test_filter_and_oc_edges(dims, radius):
    import ctypes as C

    damp = 0.5 if radius < 3 else 0.8
    ctx, G, eact, rho, vfix, r = _hier(*dims, seed=5, design_step=0.03, damp_ratio=damp)
    nx, ny, nz = dims
    act = G[0].getEact()
    sens = -np.exp(r.standard_normal(rho.size)).astype(np.float32)
    sens[r.random(rho.size) < 0.05] *= -1
    G[0].setSens(sens)
    G[0].filterSensitivity(radius)
    fo = np.zeros_like(sens)
    O.lib().or_filter(nx, ny, nz, O.ptr(act), radius, O.ptr(sens), O.ptr(fo))
    # a tap's FP32 weight 1 - 6 t^2 + 8 t^3 - 3 t^4 is a sum of terms up to 8, contracted on one side: up to 4 roundings
    # of 2^-24 x 8 = 2e-6; the weights add up to at least 1 (the centre's), and the errors of the taps rarely add
    assert rel_err(G[0].getSens(), fo) < 1e-5
    goal = float(rho.mean()) - 0.005
    G[0].setSens(fo)
    lam, trials, it = C.c_float(), C.c_int(), np.zeros(1, np.int32)
    rb._capi.check(rb.lib().rt_oc_update(G.handle, goal, C.byref(lam), C.byref(trials)), ctx.handle)
    ro, tmp = rho.ravel().copy(), np.zeros(rho.size, np.float32)
    lo = O.lib().or_oc_update(ro.size, O.ptr(act), None, O.ptr(ro), O.ptr(fo), goal, 0.03, damp, 1e-3, int(act.sum()),
                              O.ptr(it), O.ptr(tmp))
    # a power rounded differently moves the volume by 1e-7; the bisection stops at 1e-4 of it
    assert np.abs(G[0].getRho() - ro).max() <= 1e-4 and abs(lam.value - lo) <= 1e-3 * abs(lo)
    G.close()
    ctx.close()


# the blocked inverse of the coarsest matrix: n = 3 (nodes) below, at and above multiples of its 32-column blocks,
# against the solve of the assembled matrix
@pytest.mark.parametrize("dims,limit", [((5, 4, 4), 4), ((9, 5, 4), 30), ((8, 8, 4), 60), ((31, 17, 9), 100),
                                        ((40, 24, 24), 400)])
def test_coarsest_inverse_block_edges(dims, limit):
    ctx, G, eact, rho, vfix, r = _hier(*dims, seed=2, coarsest_elements=limit)
    G.update_stencil()
    g = G[G.n_grid() - 1]
    nv, vx, vy, vz = g.nv, g.nx + 1, g.ny + 1, g.nz + 1
    st = g.getStencil().reshape(27, 3, 3, vz, vy, vx)
    A = np.zeros((nv, 3, nv, 3))
    ids = np.arange(nv).reshape(vz, vy, vx)
    for k in range(27):
        d = (k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1)
        a = tuple(slice(max(0, -s), n - max(0, s)) for s, n in zip(d, (vz, vy, vx)))
        b = tuple(slice(max(0, s), n - max(0, -s)) for s, n in zip(d, (vz, vy, vx)))
        i, j = ids[a].ravel(), ids[b].ravel()
        A[i, :, j, :] = st[(k, slice(None), slice(None)) + a].reshape(3, 3, -1).transpose(2, 0, 1)
    A = A.reshape(3 * nv, 3 * nv)
    f = r.standard_normal((3, nv))
    want = np.linalg.solve(A, f.T.ravel()).reshape(nv, 3).T
    g.setForce(f.ravel())
    g.solve_fem_host()
    got = g.getDisplacement().reshape(3, nv)
    # two FP64 inversions differ by about eps cond(A)
    assert np.abs(got - want).max() <= 1e-14 * np.linalg.cond(A) * np.abs(want).max() + 1e-12 * np.abs(want).max()
    G.close()
    ctx.close()


# sensitivity: columns of 32 x 4 elements, z-chunks of 2 to 16 layers whose next layer is loaded ahead
@pytest.mark.parametrize("nx,ny,nz", [(31, 5, 8), (32, 4, 9), (33, 9, 17), (65, 41, 33)])
def test_sensitivity_edges(nx, ny, nz):
    ctx, G, H, r = _perforated(nx, ny, nz, nx, True)
    rho = G[0].getRho()
    u = r.standard_normal(3 * G[0].nv)
    G[0].setDisplacement(u)
    rb._capi.check(rb.lib().rt_sensitivity(G.handle, 0), ctx.handle)
    want = np.zeros(nx * ny * nz, np.float32)
    O.lib().or_sensitivity(nx, ny, nz, O.ptr(H.arrs[0]["eact"]), O.ptr(rho), float(P), O.ptr(H.KE), O.ptr(u), O.ptr(want))
    # FP32 results: powf to 2 units in the last place, a product and the rounding of either side
    assert np.all(np.abs(G[0].getSens() - want) <= 6 * 2.0**-24 * np.abs(want))
    G.close()
    ctx.close()


# Galerkin stencils: 32 x 2 nodes per block (33 and 34 coarse nodes in x, odd rows), both coarsening ratios, fixed
# nodes inside and on the faces; dyadic levels below
@pytest.mark.parametrize("dims,skip", [((127, 9, 7), 1), ((131, 6, 13), 1), ((63, 7, 6), 0), ((20, 18, 14), 0)])
def test_galerkin_edges(dims, skip):
    ctx, G, eact, rho, vfix, r = _hier(*dims, seed=11, skip=skip)
    vfix[r.random(vfix.shape) < 0.01] = 1
    G.set_support(vfix)
    G.update_stencil()
    H = O.Hierarchy(eact, rho, vfix, p=P, E=E, nu=NU, skip=bool(skip))
    H.set_weights(G[0].getPenalty())
    H.update_stencil()
    for i in range(1, H.nlev):
        assert rel_err(G[i].getStencil(), H.arrs[i]["st"]) < 1e-11, f"level {i}"
    G.close()
    ctx.close()


# the two coarsest levels of an FP32 cycle in one cluster launch: 8 lanes per node up to 1280 nodes (672, 1224), 4 up
# to 2560 (1440, 1710, 2420), both parities of the sweep counts, odd sides
@pytest.mark.parametrize("dims,skip,pre,post,cs", [((21, 13, 11), 0, 2, 2, 8), ((21, 13, 11), 0, 1, 3, 0),
                                                   ((32, 16, 14), 0, 3, 1, 0), ((33, 17, 14), 0, 2, 2, 1),
                                                   ((38, 20, 20), 0, 2, 1, 0), ((70, 33, 30), 1, 2, 2, 3)])
@pytest.mark.parametrize("sup", [True, False])
@pytest.mark.parametrize("jacobi", [False, True])
def test_tail_cycle_edges(dims, skip, pre, post, cs, sup, jacobi):
    ctx, G, H, r = _perforated(*dims, sum(dims), sup, skip)
    params = G.params
    params.smoother = rb.SMOOTH_JACOBI if jacobi else rb.SMOOTH_CHEBY
    params.pre_sweeps, params.post_sweeps, params.coarse_sweeps, params.jacobi_omega = pre, post, cs, 0.5
    act = np.tile(G[0].getVact(), 3).astype(bool)
    b = r.standard_normal(3 * G[0].nv) * act
    if sup:
        b[np.tile(H.arrs[0]["vfix"], 3).astype(bool)] = 0
    else:
        Ru = np.zeros(6 * b.size)
        O.lib().or_rigid_nodes(H.lv(0), O.ptr(Ru))
        O.lib().or_displacement_project(b.size // 3, O.ptr(Ru), O.ptr(b))
    x = {}
    for prec in (rb.FP64, rb.FP32):
        params.precision = prec
        G.set_params(params)
        G.update_stencil()
        G[0].setForce(b)
        G[0].reset_displacement()
        if prec == rb.FP32:
            ctx.profile(True)
            ctx.profile_reset()
        G.pcg(1e-14, 1)
        if prec == rb.FP32:
            assert "tail_cycle_f32" in ctx.profile_stats()
            ctx.profile(False)
        x[prec] = G[0].getDisplacement()
    # one preconditioned step in FP32 against FP64: 81 terms a row x 40 steps x 2^-24, of values up to 5 times the result
    assert rel_err(x[rb.FP32], x[rb.FP64]) < 1e-3
    G.close()
    ctx.close()


# stencil levels, 32 nodes per block: 672, 2310, 462 and 540 nodes (remainders 0, 6, 14 and 28), faces on every side
@pytest.mark.parametrize("dims", [(21, 13, 11), (39, 19, 17), (20, 12, 9), (18, 16, 10)])
@pytest.mark.parametrize("sup", [True, False])
def test_stencil_level_edges(dims, sup):
    ctx, G, H, r = _perforated(*dims, sum(dims) + 2, sup, 0)
    H.arrs[1]["st"][:] = G[1].getStencil()
    act = np.tile(G[1].getVact(), 3).astype(bool)
    u, f = r.standard_normal(3 * G[1].nv) * act, r.standard_normal(3 * G[1].nv) * act
    G[1].setDisplacement(u)
    G[1].setForce(f)
    G[1].update_residual()
    res = np.zeros_like(u)
    O.lib().or_st_residual(H.lv(1), O.ptr(u), O.ptr(f), O.ptr(res))
    assert rel_err(G[1].getResidual(), res) < 1e-12  # 81 terms a row in another order
    want, tmp = u.copy(), np.zeros_like(u)
    O.lib().or_st_jacobi(H.lv(1), O.ptr(want), O.ptr(f), 0.6, O.ptr(tmp))
    G[1].smooth(rb.SMOOTH_JACOBI, 1, 0.6)
    # the block division amplifies FP64 rounding on the 1e9-contrast stencils
    assert rel_err(G[1].getDisplacement(), want) < 1e-9
    G.close()
    ctx.close()


# elements of zero density inside the box and at a support, so that nodes are left without a weighted element: they keep
# their values, a fixed one takes 0, and the smoother bounds and solves are those of the body without these elements
@pytest.mark.parametrize("zc", [0, 3])
def test_zero_density_pocket(zc):
    nx, ny, nz = 36, 13, 11
    ctx, G, eact, rho, vfix, r = _hier(nx, ny, nz, seed=6)
    hole = np.zeros((nz, ny, nx), bool)
    hole[3:7, 4:8, 20:25] = True
    hole[2:5, 2:5, 0:3] = True  # nodes (0, 3, 3), (0, 3, 4), ... of the clamped face
    rho[hole] = 0
    G[0].setRho(rho.ravel())
    G.update_stencil()
    L = rb.lib()
    if zc:
        for prec in (rb.FP64, rb.FP32):
            for m in range(4):
                rb._capi.check(L.rt_set_tuning(G.handle, prec, m, 8, 1, zc), ctx.handle)
    live = np.zeros((nz + 1, ny + 1, nx + 1), bool)
    for z, y, x in np.argwhere(~hole):
        live[z:z + 2, y:y + 2, x:x + 2] = True
    dead, fixed = np.tile(~live.ravel(), 3), np.tile(vfix.ravel().astype(bool), 3)
    assert (dead & fixed).any() and (dead & ~fixed).any()
    # n_e of a fixed node counts weighted elements: the oracle gets the body without the others
    H = O.Hierarchy((~hole).astype(np.uint8), rho, vfix, p=P, E=E, nu=NU)
    H.set_weights(G[0].getPenalty())
    lm = [G.smoother_lmax(i) for i in range(H.nlev - 1)]
    assert np.isfinite(lm).all()
    H.set_lmax(lm)
    u, f = r.standard_normal(dead.size), r.standard_normal(dead.size)
    ujac, ucheb, tmp, d = u.copy(), np.zeros_like(u), np.zeros_like(u), np.zeros_like(u)
    O.lib().or_fine_jacobi(H.lv(0), O.ptr(H.KE), O.ptr(ujac), O.ptr(f), 0.6, O.ptr(tmp))
    O.lib().or_fine_cheby(H.lv(0), O.ptr(H.KE), O.ptr(u), O.ptr(f), O.ptr(ucheb), O.ptr(d), 0)
    keep = np.where(fixed, 0.0, u)
    G[0].setForce(f)
    for smoother, m, w in ((rb.SMOOTH_JACOBI, 2, ujac), (rb.SMOOTH_CHEBY, 3, ucheb)):
        w = np.where(dead, keep, w)
        G[0].setDisplacement(u)
        G[0].smooth(smoother, 1, 0.6)
        assert rel_err(G[0].getDisplacement(), w) < 1e-10
        G[0].setDisplacement(u)
        rb._capi.check(L.rt_fine_kernel_f32(G.handle, m, 0.6), ctx.handle)
        assert rel_err(G[0].getResidual(), w) < 2e-6
    # the same body with the elements taken out
    ctx2, G2, *_ = _hier(nx, ny, nz, seed=6)
    G2.close()
    G2 = rb.HierarchyGrid(ctx2, G.params)
    G2.genFromBox((~hole).astype(np.uint8))
    G2[0].setRho(rho.ravel())
    G2.set_support(vfix)
    b = f * ~dead * ~fixed
    for form in (dict(precision=rb.FP64, smoother=rb.SMOOTH_JACOBI, jacobi_omega=0.5),
                 dict(precision=rb.FP32, smoother=rb.SMOOTH_CHEBY)):
        x = []
        for g in (G, G2):
            p = g.params
            p.pre_sweeps = p.post_sweeps = 2
            for k, v in form.items():
                setattr(p, k, v)
            g.set_params(p)
            g.update_stencil()
            g[0].setForce(b)
            g[0].reset_displacement()
            assert g.pcg(1e-9, 500).rel_residual <= 1e-9
            x.append(g[0].getDisplacement())
        assert abs(G.smoother_lmax(0) - G2.smoother_lmax(0)) < 1e-9 * G2.smoother_lmax(0)
        # two solves to 1e-9 of the residual, amplified by the condition of the 1e3-contrast body; the coarse levels'
        # corrections leave any values in the nodes without stiffness
        assert rel_err(x[0][~dead], x[1][~dead]) < 1e-4
    G2.close()
    ctx2.close()
    G.close()
    ctx.close()


# FP32 block inverse of the finest level: formed in FP64 and rounded once, so that a step from u = 0 has the rounding of
# its entries and of the result alone, also where a product of three entries of the block leaves FP32's range
@pytest.mark.parametrize("scale,lo", [(1.0, 0.1), (1e8, 0.1), (1e-8, 1e-3)])
def test_fp32_block_inverse(scale, lo):
    nx, ny, nz = 37, 15, 12
    ctx, G, eact, rho, vfix, r = _hier(nx, ny, nz, seed=8)
    p = G.params
    p.youngs_modulus = E * scale
    G.set_params(p)
    rho = (lo * 10.0 ** (r.random(eact.shape) * -np.log10(lo))).astype(np.float32)
    G[0].setRho(rho.ravel())
    f = r.standard_normal(3 * G[0].nv).astype(np.float32).astype(np.float64)
    G[0].setForce(f)
    G[0].reset_displacement()
    G[0].update_residual()
    H = O.Hierarchy(eact, rho, vfix, p=P, E=E * scale, nu=NU)
    H.set_weights(G[0].getPenalty())
    want, tmp = np.zeros_like(f), np.zeros_like(f)
    O.lib().or_fine_jacobi(H.lv(0), O.ptr(H.KE), O.ptr(want), O.ptr(f), 1.0, O.ptr(tmp))
    rb._capi.check(rb.lib().rt_fine_kernel_f32(G.handle, 2, 1.0), ctx.handle)
    got = G[0].getResidual()
    n = G[0].nv
    err = np.abs(got - want).reshape(3, n).max(0) / np.abs(want).reshape(3, n).max(0)
    # entries, products and sums to 2^-24, the products at most twice the result (condition of the block): 4 units at most
    assert err.max() < 4 * 2.0**-24, err.max() * 2.0**24
    G.close()
    ctx.close()


# the stored FP32 blocks are there and current whichever call first needs them: a launch shape chosen after the stencils,
# a density change, a workspace's smoothing right after new supports
def test_fp32_blocks_follow():
    L = rb.lib()
    ctx, G, eact, rho, vfix, r = _hier(33, 17, 14, seed=9, precision=rb.FP32, smoother=rb.SMOOTH_CHEBY, pre_sweeps=2,
                                       post_sweeps=2)
    b = r.standard_normal(3 * G[0].nv) * np.tile(1.0 - vfix.ravel(), 3)

    def step(g, shape=None):
        if shape:
            g.set_tiles(*shape)
        g[0].setForce(b)
        g[0].reset_displacement()
        g.pcg(1e-14, 2)
        return g[0].getDisplacement()

    shape = G.tuning()["chebyshev_f32"]["zchunk"]
    for new in (rho, (0.1 + 0.9 * r.random(rho.shape)).astype(np.float32)):
        G[0].setRho(new.ravel())
        G.set_tiles(3, 8, 16)  # reads no blocks
        G.update_stencil()
        late = step(G, (8, 1, shape))
        G.update_stencil()
        assert np.array_equal(late, step(G))
    # a hierarchy without blocks yet, and its tuner
    G2 = rb.HierarchyGrid(ctx, G.params)
    G2.genFromBox(eact)
    G2[0].setRho(new.ravel())
    G2.set_support(vfix)
    G2.set_tiles(3, 8, 16)
    G2.update_stencil()
    assert G2.autotune(2)["chebyshev_f32"]["us"] > 0
    step(G2)
    G2.close()
    W = G.workspace()
    vfix[:, :, -1] = 1
    G.set_support(vfix)
    got = []
    for g in (W, G):
        g[0].setForce(b)
        g[0].setDisplacement(b)
        rb._capi.check(L.rt_smooth_f32(g.handle, 0, rb.SMOOTH_JACOBI, 2, 0.6), ctx.handle)
        got.append(g[0].getDisplacement())
    assert np.array_equal(*got)
    G.close()
    ctx.close()


# the finest Gauss-Seidel divides by the diagonal: from u = 0 the first colour's first component is f / (KE_00 sum w), and
# a sum of 8 FP32 weights is exact in FP64, so that any other rounding of the quotient shows
def test_fine_gauss_seidel_quotient():
    nx, ny, nz = 25, 13, 11
    ctx, G, eact, rho, vfix, r = _hier(nx, ny, nz, seed=12, sup=False)
    f = r.standard_normal((3, nz + 1, ny + 1, nx + 1))
    G[0].setForce(f.ravel())
    G[0].reset_displacement()
    G[0].smooth(rb.SMOOTH_GS, 1)
    w = np.zeros((nz + 2, ny + 2, nx + 2))
    w[1:-1, 1:-1, 1:-1] = G[0].getPenalty().reshape(nz, ny, nx)
    sw = sum(w[k:nz + 1 + k, j:ny + 1 + j, i:nx + 1 + i] for k in (0, 1) for j in (0, 1) for i in (0, 1))
    want = f[0] / (G.template_matrix().ravel()[0] * sw)
    assert np.array_equal(G[0].getDisplacement().reshape(f.shape)[0, ::2, ::2, ::2], want[::2, ::2, ::2])
    G.close()
    ctx.close()


# the FP32 step from zero with stored blocks takes a second node per thread past 32 x 256 nodes per SM: one iteration of
# either precision's cycle, whose first step that is, on a box of 1.3M nodes and supports at both its ends
@pytest.mark.parametrize("jacobi", [False, True])
def test_step_from_zero_second_node(jacobi):
    ctx, G, eact, rho, vfix, r = _hier(133, 103, 97, seed=13)
    vfix[-1] = 1
    G.set_support(vfix)
    p = G.params
    p.pre_sweeps, p.post_sweeps, p.jacobi_omega = 1, 1, 0.5
    p.smoother = rb.SMOOTH_JACOBI if jacobi else rb.SMOOTH_CHEBY
    b = r.standard_normal(3 * G[0].nv) * np.tile(1.0 - vfix.ravel(), 3)
    x = []
    for prec in (rb.FP64, rb.FP32):
        p.precision = prec
        G.set_params(p)
        G.update_stencil()
        G[0].setForce(b)
        G[0].reset_displacement()
        G.pcg(1e-14, 1)
        x.append(G[0].getDisplacement())
    # as in test_tail_cycle_edges
    assert rel_err(x[1], x[0]) < 1e-3
    G.close()
    ctx.close()
