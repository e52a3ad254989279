"""GPU kernels at the sizes where their tiles, words and runs end, bit-exact
against the CPU oracle: the filters' level images and 2 x 2 x 2 blocks (rows of
less than a word, one cell more or less than a word or a tile, rows whose words
are staged in several parts, single planes and rows, odd extents), the coarse
pulling-scheme levels, the dilations of long rows, the inverse B-spline's short
runs, the strided passes' lines per thread and the padded lines; and the
network layer's gradients over whole and partial tiles."""
import ctypes as C

import numpy as np
import pytest

import libapr_b200 as A
from libapr_b200._lib import check, lib
from oracle import bind as B
from tests.helpers import bits_equal, gaussian_psf, lib_params, oracle_params, random_stencil, volume

pytestmark = pytest.mark.gpu

# (z, x, y): words of 32 cells in y, tiles of 16 x 128 cells and 8 planes
FILTER_SHAPES = [((1, 1, 100), 3), ((1, 40, 65), 6), ((2, 17, 129), 8), ((9, 33, 128), 12), ((8, 16, 66), 6),
                 ((33, 18, 131), 20), ((17, 50, 257), 20), ((3, 3, 3), 1), ((33, 1, 34), 4), ((20, 2, 40), 5),
                 ((2, 2, 66), 2), ((5, 70, 2), 3)]


def built(shape, blobs, image_type=0, seed=11, img=None, **kw):
    img = volume(shape, blobs, seed) if img is None else img
    e, acc, _ = B.orc_get_apr(img, oracle_params(**kw), image_type)
    assert e == 0
    conv = A.APRConverter("uint16" if image_type == 1 else "float")
    conv.par = lib_params(**kw)
    apr = A.APR()
    assert conv.get_apr(apr, img)
    return img, acc, apr


@pytest.mark.parametrize("shape,blobs", FILTER_SHAPES)
def test_filters_at_edges(shape, blobs):
    check_filters(*built(shape, blobs))


@pytest.mark.parametrize("weight", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("ks", [3, 5])
def test_weights_that_are_not_finite_on_a_plane(ks, weight):
    """A stencil's taps beside a single plane are 0 times their weight: not a number
    where the weight is not finite, in float and in double."""
    img, acc, apr = built((1, 40, 65), 6)
    raw = B.orc_sample(acc, img)
    st = random_stencil(ks, 5)
    st[0] = weight
    for reflect in (True, False):
        out = A.APRFilter.convolve_pencil(apr, st, raw.astype(np.float32), reflect_boundary=reflect,
                                          use_stencil_downsample=False, normalize=False)
        assert np.isnan(out).all()
    out = A.APRNumerics.richardson_lucy(apr, raw, None, st, 1, use_stencil_downsample=False, dtype=np.float64)
    assert np.isnan(out).all()


def crossed(shape, seed):
    """A volume with a bright ridge across every y that is a multiple of 1024: rows
    stage their words 2048 cells (parents: 1024) at a time."""
    img = volume(shape, 4, seed).astype(np.int64)
    y = np.arange(shape[2])
    for c in range(1024, shape[2], 1024):
        img += (40000 * np.exp(-((y - c) / 5.0) ** 2)).astype(np.int64)
    return img.clip(0, 65535).astype(np.uint16)


# levels of 2049, 2113, of 4161 and 2081 and of 9001 - 2251 cells along y; few rows,
# so a row also goes to several warps
@pytest.mark.parametrize("shape", [(3, 5, 2049), (4, 6, 2113), (2, 3, 4161), (1, 1, 9001)])
def test_filters_on_rows_of_several_parts(shape):
    img, acc, apr = built(shape, 0, img=crossed(shape, 11))
    tree = B.orc_tree(acc)
    for a, top, part in ((acc, acc.l_max, 2048), (tree, tree.l_max, 1024)):
        lev, z, x, y = a.particle_coords()
        for l in range(a.l_min, top + 1):  # elements at both sides of the parts' edge
            if a.y_num[l] > part + 1:
                d = y[lev == l].astype(int) - part
                assert ((d >= -8) & (d < 0)).any() and ((d >= 0) & (d < 8)).any(), l
    check_filters(img, acc, apr)


def check_filters(img, acc, apr):
    tr = B.orc_tree(acc)
    raw = B.orc_sample(acc, img)
    parts = raw.astype(np.float32)
    assert bits_equal(A.APRTreeNumerics.fill_tree_mean(apr, parts), B.orc_tree_mean(acc, tr, parts))
    for ks in (3, 5):
        st = random_stencil(ks, 300 + ks)
        for reflect in (True, False):
            ref, _ = B.orc_convolve(acc, tr, st, parts, reflect=reflect, use_stencil_ds=True, normalize=False)
            out = A.APRFilter.convolve_pencil(apr, st, parts, reflect_boundary=reflect)
            assert bits_equal(out, ref), (ks, reflect)
    deltas = (1.0, 0.5, 2.0)
    for sobel, fn in ((False, A.APRNumerics.gradient_magnitude_cfd), (True, A.APRNumerics.gradient_magnitude_sobel)):
        assert bits_equal(fn(apr, parts, deltas), B.orc_gradient(acc, tr, parts, -1, sobel, deltas)), sobel
    psf = gaussian_psf()
    ref = B.orc_richardson_lucy(acc, tr, raw, psf, 2, normalize=True, use_double=True)
    out = A.APRNumerics.richardson_lucy(apr, raw, None, psf, 2, normalize=True, dtype=np.float64)
    assert np.array_equal(out.view(np.uint64), ref.view(np.uint64))


def test_level_image_in_runs_of_planes():
    """A level whose image exceeds the scratch of one run (67 MB a plane: runs of
    8 planes at 3^3) gives the bits of the same call in place, which builds the
    whole level's image at once."""
    import torch
    img = torch.empty(20, 2048, 8192, dtype=torch.int16, device="cuda")
    A.synth_blobs_device(img, 2000, seed=5)
    conv = A.APRConverter("float")
    conv.par = lib_params()
    apr = A.APR()
    assert conv.get_apr(apr, img)
    n = apr.total_number_particles()
    x = torch.empty(n, device="cuda").uniform_(0, 1000)
    st = np.ascontiguousarray(random_stencil(3, 7).ravel())
    y = torch.empty_like(x)
    for dst in (y, x):
        check(lib().aprb_convolve_device(apr._h, st.ctypes.data_as(C.c_void_p), 3, C.c_void_p(x.data_ptr()),
                                         C.c_void_p(dst.data_ptr()), 1, 1, 0, None))
    assert torch.equal(x.view(torch.int32), y.view(torch.int32))


# l_max 2 .. 9 (levels up to 5 run in one CTA), odd and unequal extents
@pytest.mark.parametrize("shape,blobs", [((4, 3, 4), 1), ((3, 5, 9), 1), ((16, 16, 16), 3), ((17, 33, 29), 8),
                                         ((32, 32, 32), 10), ((40, 20, 70), 12), ((5, 70, 3), 2), ((66, 64, 65), 30),
                                         ((3, 6, 400), 3)])
@pytest.mark.parametrize("nopt", [True, False])
def test_structure_of_coarse_levels(shape, blobs, nopt):
    img, acc, apr = built(shape, blobs, seed=13, neighborhood_optimization=nopt)
    lx, xe, yv = apr.linear_access()
    assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)
    assert np.array_equal(A.ParticleData().sample_image(apr, img).data, B.orc_sample(acc, img))


# levels whose rows (513 - 1050 cells, not a multiple of 16) take several CTAs of a
# dilation along y
@pytest.mark.parametrize("shape,blobs", [((5, 9, 1026), 12), ((20, 17, 1030), 40), ((9, 40, 1061), 60),
                                         ((3, 5, 2100), 30)])
def test_structure_of_long_rows(shape, blobs):
    img, acc, apr = built(shape, blobs, seed=29)
    lx, xe, yv = apr.linear_access()
    assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)


# z lines 160000 (four per thread), 90000 (two), 65536 (one); the x lines are few
@pytest.mark.parametrize("shape", [(6, 400, 400), (8, 300, 300), (8, 256, 256), (5, 302, 301)])
@pytest.mark.parametrize("image_type", [0, 1])
def test_strided_passes_lines_per_thread(shape, image_type):
    img, acc, apr = built(shape, 20, image_type, seed=17)
    lx, xe, yv = apr.linear_access()
    assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)


def gradient_runs(geo):
    """Runs of 32 cells for which the input gradient's stencil has nothing to do (no
    particle of the level within one cell), those of them that start inside a word
    of 32 cells, and runs that only a particle next to them keeps."""
    skipped = inside = beside = 0
    for l in range(geo.acc.l_min, geo.acc.l_max + 1):
        zn, xn, yn = geo.dims(l)
        m = geo.plev == l
        if not m.any():
            continue
        held = np.zeros((zn + 2, xn + 2, yn + 2), bool)
        held[geo.pz[m] + 1, geo.px[m] + 1, geo.py[m] + 1] = True
        for k in range(0, zn * xn * yn, 32):
            z, x, y = k // yn // xn, k // yn % xn, k % yn
            if y + 32 > yn:
                continue
            near = held[z:z + 3, x:x + 3, y:y + 34]
            if not near.any():
                skipped += 1
                inside += y % 32 != 0
            elif not near[1, 1, 1:33].any():
                beside += 1
    return skipped, inside, beside


@pytest.mark.parametrize("shape,blobs", [((8, 8, 9), 1), ((12, 20, 33), 4), ((9, 14, 150), 2), ((5, 12, 197), 2),
                                         ((6, 40, 97), 2)])
def test_network_gradients_over_tiles(shape, blobs):
    """The weight and bias gradients add up over whole and partial tiles of 16
    particles on every level, and the input gradient skips nothing that a particle
    reaches.  Operands are small integers and their tree means, eighths of eighths,
    which 32 bits and so both sides' roundings to bfloat16 hold alike; what is left
    is the rounding of sums, 2^-23 of the sum of magnitudes for each addition."""
    import torch
    img, acc, apr = built(shape, blobs)
    from oracle import cnn_oracle as O
    geo = O.Geometry(acc, B.orc_tree(acc))
    if shape[2] >= 97:  # sparse enough for the skip, at many offsets
        assert min(gradient_runs(geo)) >= 10
    rng = np.random.default_rng(2)
    H = rng.integers(-2, 3, size=(geo.P, 16)).astype(np.float32)
    G = rng.integers(-2, 3, size=(geo.P, 16)).astype(np.float32)
    W = rng.integers(-1, 2, size=(27, 16, 16)).astype(np.float32)
    H64, W64, G64 = (a.astype(np.float64) for a in (H, W, G))
    ref_in, ref_dW, ref_db = O.layer_backward(geo, H64, W64, None, G64, False, round_bf16=True)
    mag_in, mag_dW, _ = O.layer_backward(geo, abs(H64), abs(W64), None, abs(G64), False, round_bf16=True)
    # dW: the 17 additions of a step for up to nine steps a CTA, then one addition a CTA on every level
    bound_dW = 2.0 ** -23 * (9 * 17 + geo.P // 16 + acc.l_max + 1) * mag_dW
    bound_in = 2.0 ** -23 * 2 * (acc.l_max + 1) * mag_in  # cells and parents are integers; one addition a tree level
    one = G64.copy()
    one[np.nonzero(geo.plev == acc.l_max)[0][-1]] = 0  # the bound sees a single particle left out
    assert (abs(O.layer_backward(geo, H64, W64, None, one, False, round_bf16=True)[1] - ref_dW) > bound_dW).any()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    h, w, g = dev(H), dev(W), dev(G)
    g_in, dW, db = torch.empty_like(h), torch.zeros_like(w), torch.zeros(16, device="cuda")
    p = A.learned._p
    check(lib().aprb_cnn_layer_backward_device(apr._h, p(h), p(w), p(h), p(g), 0, p(g_in), p(dW), p(db), None))
    assert np.array_equal(db.cpu().numpy(), ref_db.astype(np.float32))
    assert np.all(abs(dW.cpu().numpy() - ref_dW) <= bound_dW)
    assert np.all(abs(g_in.cpu().numpy() - ref_in) <= bound_in)


# the blocked converter's level images and seeds, tile by tile: one CTA for the
# levels of up to 16 cells, single planes and ghosts at both ends
@pytest.mark.parametrize("shape,zb,ghost", [((40, 70, 33), 8, 4), ((100, 20, 130), 32, 16), ((9, 5, 6), 4, 2),
                                            ((64, 257, 30), 16, 2)])
def test_block_patches(shape, zb, ghost):
    img = volume(shape, 12, 23)
    e, acc = B.orc_get_apr_by_block(img, oracle_params(), 0, zb, ghost)
    assert e == 0
    conv = A.APRConverterBatch("float", z_block_size=zb, ghost_z=ghost)
    conv.par = lib_params()
    apr = A.APR()
    assert conv.get_apr(apr, img)
    lx, xe, yv = apr.linear_access()
    assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)


def test_pyramid_solved_by_a_converter_that_filled_no_tile():
    """A uint16 APR records the offset of the image it was made from, which only a
    converter that filled a tile knows: the call is refused.  Float images have none."""
    import torch
    from libapr_b200.distributed import TileBackend, tile_count
    shape, zb, ghost = (40, 70, 33), 8, 4
    img = volume(shape, 12, 23)
    slab = torch.from_numpy(img.view(np.int16)).cuda()
    for image_type, name in ((1, "uint16"), (0, "float")):
        fill, solve = TileBackend(name, lib_params()), TileBackend(name, lib_params())
        pyr = fill.pyramid(shape)
        fill.fill(pyr, shape, zb, ghost, 0, tile_count(shape[0], zb), slab, 0)
        if image_type == 1:
            with pytest.raises(RuntimeError, match="offset"):
                solve.finish(pyr, shape)
            apr = fill.finish(pyr, shape)
        else:
            apr = solve.finish(pyr, shape)
            assert apr.bspline_offset() == 0
        e, acc = B.orc_get_apr_by_block(img, oracle_params(), image_type, zb, ghost)
        assert e == 0
        lx, xe, yv = apr.linear_access()
        assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)


# rows of 4k + 1 .. 4k + 3 samples of a megavoxel or more: lines padded to a
# multiple of 8 (float ImageType), every stage compared
@pytest.mark.parametrize("shape", [(64, 130, 129), (33, 250, 130), (17, 260, 259), (40, 100, 267), (1, 4100, 257)])
def test_padded_lines(shape):
    img = volume(shape, 30, 19)
    e, acc, (off, inter) = B.orc_get_apr(img, oracle_params(), 0)
    assert e == 0
    conv = A.APRConverter("float")
    conv.par = lib_params()
    conv.keep_intermediates(True)
    import torch
    apr = A.APR()
    assert conv.get_apr(apr, torch.from_numpy(img.view(np.int16)).cuda())
    assert bits_equal(conv.intermediate(0, shape), inter[0])
    ds = tuple((n + 1) // 2 for n in shape)
    for w in range(1, 7):
        assert bits_equal(conv.intermediate(w, ds), inter[w]), w
    lx, xe, yv = apr.linear_access()
    assert np.array_equal(xe, acc.xz_end) and np.array_equal(yv, acc.y_vec)



# padded in two runs of 2^26 samples: 815 and 5 lines past the first run's; the
# host-buffer call does not pad its lines
@pytest.mark.parametrize("shape", [(130, 999, 517), (180, 717, 517)])
def test_padded_lines_in_runs(shape):
    import torch
    img = torch.empty(*shape, dtype=torch.int16, device="cuda")
    A.synth_blobs_device(img, 2000, seed=31)
    first = (1 << 26) // 520
    assert first < shape[0] * shape[1] and (shape[0] * shape[1] - first < 32) == (shape[1] == 717)
    aprs, smooth = [], []
    for src in (img, img.cpu().numpy().view(np.uint16)):
        conv = A.APRConverter("float")
        conv.par = lib_params()
        conv.keep_intermediates(True)
        apr = A.APR()
        assert conv.get_apr(apr, src)
        smooth.append(conv.intermediate(0, shape))
        aprs.append(apr.linear_access())
        del conv
    assert bits_equal(*smooth)
    for a, b in zip(*aprs):
        assert np.array_equal(a, b)
