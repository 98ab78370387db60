"""The kernels for many rows (one, two or four warps per row) against the one-CTA-per-row kernels on the same rows in smaller
calls: the same bits, at partial slices, partial CTAs and both sides of the row threshold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP = 384      # rows per small call: below every threshold (up to 8191 columns), whole scale-factor atoms


def _dev(a):
    from gpu_util import Dev
    return Dev(a)


def _rows(seed, rows, dim):
    from gpu_util import rand_bf16
    x = rand_bf16(np.random.default_rng(seed), (rows, dim))
    x[3, : dim // 2] = 0
    x[5] = 0x8000                                            # a row of -0
    x[7, 16:32] = 0x4300
    return x


@pytest.mark.parametrize("rows,dim", [(1536, 1024), (3075, 776), (3073, 2064), (3072, 4096), (1539, 3072)])
@pytest.mark.parametrize("kind", ["fp8", "bf16", "nvfp4_0", "nvfp4_1"])
def test_norm_rows(rows, dim, kind):
    from flashrt_b200 import _lib
    from gpu_util import f32, rand_bf16, zeros
    if kind.startswith("nvfp4"):
        rows, dim = max(rows, 3072), dim // 16 * 16
    x = _rows(rows + dim, rows, dim)
    w = _dev(rand_bf16(np.random.default_rng(1), (dim,)))
    sc, got = f32(0.011), []
    katoms = (dim + 63) // 64
    for step in (rows, STEP):
        d_x, d_o = _dev(x), zeros((rows, dim * (2 if kind == "bf16" else 1)), np.uint8)
        d_sf = zeros(((rows + 127) // 128 * katoms * 512,), np.uint8)
        for r in range(0, rows, step):
            n = min(step, rows - r)
            xp = d_x.ptr + r * dim * 2
            if kind == "fp8":
                _lib.call("frt_b200_norm_fp8", xp, None, None, 0, w.ptr, None, 0, d_o.ptr + r * dim, None, n, dim, 1e-6, sc.ptr, 0, 0)
            elif kind == "bf16":
                _lib.call("frt_b200_norm_bf16", xp, None, None, 0, None, None, 0, d_o.ptr + r * dim * 2, None, n, dim, 1e-6, 0, 0)
            else:
                _lib.call("frt_b200_norm_nvfp4", xp, None, None, 0, w.ptr, None, 0, d_o.ptr + r * dim // 2,
                          d_sf.ptr + r // 128 * katoms * 512, None, n, dim, 1e-6, int(kind[-1]), 0, 0)
        got.append((d_o.get(), d_sf.get()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("rows,dim", [(1024, 3072), (1027, 520), (1025, 4104)])
@pytest.mark.parametrize("mod", ["affine", "modulated", "plain"])
def test_layer_norm_rows_and_residual_form(rows, dim, mod):
    """Also the residual update in the same pass against bias_gate_mul_residual / residual_add, then layer_norm."""
    from flashrt_b200 import _lib, flash_rt_kernels as fvk
    from gpu_util import f32, rand_bf16, zeros
    rng = np.random.default_rng(rows + dim)
    x, y = _rows(2, rows, dim), rand_bf16(rng, (rows, dim))
    w, b, sc, sh, gate = (_dev(rand_bf16(rng, (2, dim))) for _ in range(5))
    aff = (w.ptr, b.ptr) if mod == "affine" else (None, None)
    md = (sc.ptr, sh.ptr) if mod == "modulated" else (None, None)
    s8, outs = f32(0.013), []
    for step in (rows, STEP):
        d_x, d_o = _dev(x), zeros((rows, dim), np.uint8)
        for r in range(0, rows, step):
            _lib.call("frt_b200_layer_norm", d_x.ptr + r * dim * 2, *aff, *md, 0, d_o.ptr + r * dim, None, s8.ptr,
                      min(step, rows - r), dim, 1e-6, 0, 0)
        outs.append(d_o.get())
    assert np.array_equal(outs[0], outs[1])
    # two modulation rows, the second from row `half` on
    half = rows // 2 + 1
    for g in (gate.ptr, 0):
        d_x, d_y, d_o = _dev(x), _dev(y), zeros((rows, dim), np.uint8)
        d_r, d_o2 = zeros((rows, dim), np.uint16), zeros((rows, dim), np.uint8)
        fvk.residual_layer_norm_fp8(d_x.ptr, d_y.ptr, g, d_r.ptr, d_o2.ptr, s8.ptr, rows, dim, 1e-6, 0, weight=aff[0] or 0,
                                    bias=aff[1] or 0, scale=md[0] or 0, shift=md[1] or 0, mod_stride=dim, mod_rows=half)
        for i, (r, n) in enumerate(((0, half), (half, rows - half))):
            o = r * dim * 2
            if g:
                fvk.bias_gate_mul_residual_bf16(d_x.ptr + o, d_y.ptr + o, 0, g + i * dim * 2, n, dim, 0, gate_stride=0)
            else:
                fvk.residual_add(d_x.ptr + o, d_y.ptr + o, n * dim, 0)
            _lib.call("frt_b200_layer_norm", d_x.ptr + o, *aff, *(p + i * dim * 2 if p else None for p in md), 0,
                      d_o.ptr + r * dim, None, s8.ptr, n, dim, 1e-6, 0, 0)
        assert np.array_equal(d_r.get() & 0x7fff, d_x.get() & 0x7fff)          # up to the sign of zeros
        assert np.array_equal(d_o.get(), d_o2.get())


@pytest.mark.parametrize("dims,lines,res_lines", [((520, 1024), (8, 20), (6, 20, 80)), ((1032, 1536), (6, 8, 14, 16), (28,)),
                                                  ((1800, 2048), (5, 10, 15, 20, 40), (80,)), ((2056, 2560), (5, 8, 10, 16, 30), (8, 10, 30)),
                                                  ((2568, 3072), (3, 8, 10, 16, 40), (8, 10, 30))])
@pytest.mark.parametrize("mod", ["affine", "modulated"])
def test_layer_norm_at_the_lines_between_kernels(dims, lines, res_lines, mod):
    """`lines` rows per SM are where another kernel takes over: one row more than that many, against the same rows in calls of 128
    (one CTA per row; with the residual the form for few rows): the same bits.  FP8, bf16 and the residual form."""
    import torch
    from flashrt_b200 import _lib
    from gpu_util import f32, rand_bf16, zeros
    sms, rng = torch.cuda.get_device_properties(0).multi_processor_count, np.random.default_rng(dims[0])
    s8 = f32(0.013)
    for dim in dims:
        vec = [_dev(rand_bf16(rng, (dim,))) for _ in range(3)]
        aff, md = ((vec[0].ptr, vec[1].ptr), (None, None)) if mod == "affine" else ((None, None), (vec[0].ptr, vec[1].ptr))
        top = sms * max(lines + res_lines) + 1
        d_x, d_y = _dev(_rows(dim, top, dim)), _dev(_rows(dim + 1, top, dim))
        for kind, per_sm in [(k, n) for k in ("fp8", "bf16") for n in lines] + [("res", n) for n in res_lines]:
            rows, outs = per_sm * sms + 1, []
            for step in (rows, 128):
                d_o = torch.zeros(rows, dim, dtype=torch.uint16 if kind == "bf16" else torch.uint8, device="cuda")
                d_r = torch.zeros(rows, dim, dtype=torch.uint16, device="cuda")
                for r in range(0, rows, step):
                    n, xp, yp, op = min(step, rows - r), d_x.ptr + r * dim * 2, d_y.ptr + r * dim * 2, d_o[r:].data_ptr()
                    if kind == "res":
                        _lib.call("frt_b200_residual_layer_norm_fp8", xp, yp, vec[2].ptr, d_r[r:].data_ptr(), *aff, *md, 0, n, op,
                                  s8.ptr, n, dim, 1e-6, 0, 0)
                    else:
                        _lib.call("frt_b200_layer_norm", xp, *aff, *md, 0, op if kind == "fp8" else None,
                                  op if kind == "bf16" else None, s8.ptr, n, dim, 1e-6, 0, 0)
                torch.cuda.synchronize()
                outs.append((d_o.view(torch.uint8), d_r.view(torch.uint8)))
            assert all(torch.equal(g, w) for g, w in zip(*outs)), (dim, kind, per_sm)


@pytest.mark.parametrize("L,heads,hd,seq", [(512, 24, 128, 512), (515, 3, 40, 400), (513, 5, 256, 513)])
def test_qkv_split_norm_rope_rows(L, heads, hd, seq):
    from flashrt_b200 import flash_rt_kernels as fvk
    from gpu_util import rand_bf16, zeros
    rng = np.random.default_rng(L)
    dim = heads * hd
    qkv, wq, wk = _dev(rand_bf16(rng, (L, 3 * dim))), _dev(rand_bf16(rng, (dim,))), _dev(rand_bf16(rng, (dim,)))
    fr, fi = (_dev(rng.standard_normal((L, hd // 2)).astype(np.float32)) for _ in range(2))
    outs = []
    for step in (L, 256):
        q, k = zeros((L, dim), np.uint16), zeros((L, dim), np.uint16)
        for r in range(0, L, step):
            n = min(step, L - r)
            o = r * hd // 2 * 4
            fvk.qkv_split_norm_rope_bf16(qkv.ptr + r * 3 * dim * 2, wq.ptr, wk.ptr, fr.ptr + o, fi.ptr + o, q.ptr + r * dim * 2,
                                         k.ptr + r * dim * 2, 1, n, heads, hd, max(0, min(n, seq - r)), 1e-6, 0)
        outs.append((q.get(), k.get()))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("rows,dim", [(3073, 1024), (3077, 1040), (1027, 3072), (1111, 3088), (769, 4112), (389, 8192)])
@pytest.mark.parametrize("kind", ["fp8", "nvfp4_0", "nvfp4_1"])
def test_norm_blocks_of_unaligned_rows(rows, dim, kind):
    """One, two and four warps per row: the last piece of a row partly there, rows and results that start 16 (8) bytes off the
    widest access, values of every class."""
    from flashrt_b200 import _lib
    from gpu_util import f32, rand_bf16, zeros
    x = _rows(rows + dim, rows, dim)
    x[9, 3], x[11, 17], x[13, 40:48] = 0x7f80, 0x7fc0, 0x0001      # inf, NaN, subnormal values
    w, sc, katoms, got = _dev(rand_bf16(np.random.default_rng(1), (dim,))), f32(0.011), (dim + 63) // 64, []
    buf = np.zeros(rows * dim + 8, np.uint16)
    for off, step in ((0, rows), (8, rows), (0, 256)):
        buf[off:off + rows * dim] = x.reshape(-1)
        d_x, d_o, d_sf = _dev(buf), zeros((rows * dim + 8,), np.uint8), zeros(((rows + 127) // 128 * katoms * 512,), np.uint8)
        for r in range(0, rows, step):
            n, xp = min(step, rows - r), d_x.ptr + (r * dim + off) * 2
            if kind == "fp8":
                _lib.call("frt_b200_norm_fp8", xp, None, None, 0, w.ptr, None, 0, d_o.ptr + r * dim + off, None, n, dim, 1e-6,
                          sc.ptr, 0, 0)
            else:
                _lib.call("frt_b200_norm_nvfp4", xp, None, None, 0, w.ptr, None, 0, d_o.ptr + r * dim // 2 + off,
                          d_sf.ptr + r // 128 * katoms * 512, None, n, dim, 1e-6, int(kind[-1]), 0, 0)
        got.append((d_o.get()[off:off + rows * dim // (1 if kind == "fp8" else 2)], d_sf.get()))
    for g in got[:2]:
        assert np.array_equal(g[0], got[2][0]) and np.array_equal(g[1], got[2][1])


@pytest.mark.parametrize("dim", [520, 784, 1032, 1536, 2048, 2560, 3072])
@pytest.mark.parametrize("per_sm", [12, 14, 15, 16, 20, 40])
@pytest.mark.parametrize("kind", ["fp8", "bf16", "nvfp4_0", "nvfp4_1"])
def test_norm_rows_at_the_lines_between_kernels(dim, per_sm, kind):
    """`per_sm` rows per SM are where another kernel takes over: that many rows and one more, results on and off the widest store,
    against the same rows in calls of 256 (the one-CTA-per-row kernel): the same bits."""
    import torch
    from flashrt_b200 import _lib
    from gpu_util import f32, rand_bf16, zeros
    last = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    dim = dim // 16 * 16 if kind.startswith("nvfp4") else dim
    x = _rows(dim + per_sm, last + 1, dim)
    x[9, 3], x[11, 17], x[13, 40:48] = 0x7f80, 0x7fc0, 0x0001      # inf, NaN, subnormal values
    d_x, w, sc, katoms = _dev(x), _dev(rand_bf16(np.random.default_rng(1), (dim,))), f32(0.011), (dim + 63) // 64
    item = {"fp8": 2, "bf16": 4}.get(kind, 1)                       # half bytes per value
    got = []
    for rows, off, step in ((last + 1, 0, last + 1), (last + 1, 16, last + 1), (last, 0, last), (last + 1, 0, 256)):
        d_o, d_sf = zeros((rows * dim * item // 2 + 16,), np.uint8), zeros(((rows + 127) // 128 * katoms * 512,), np.uint8)
        off = off // (1 if kind == "bf16" else 2)                   # the least alignment the entry points take
        for r in range(0, rows, step):
            n, xp, op = min(step, rows - r), d_x.ptr + r * dim * 2, d_o.ptr + off + r * dim * item // 2
            if kind == "fp8":
                _lib.call("frt_b200_norm_fp8", xp, None, None, 0, w.ptr, None, 0, op, None, n, dim, 1e-6, sc.ptr, 0, 0)
            elif kind == "bf16":
                _lib.call("frt_b200_norm_bf16", xp, None, None, 0, w.ptr, None, 0, op, None, n, dim, 1e-6, 0, 0)
            else:
                _lib.call("frt_b200_norm_nvfp4", xp, None, None, 0, w.ptr, None, 0, op, d_sf.ptr + r // 128 * katoms * 512, None, n,
                          dim, 1e-6, int(kind[-1]), 0, 0)
        got.append((d_o.get()[off:off + last * dim * item // 2], d_o.get()[off + last * dim * item // 2:][:dim * item // 2],
                    d_sf.get()[: last // 128 * katoms * 512], rows))
    for g in got[:3]:
        assert np.array_equal(g[0], got[3][0]) and np.array_equal(g[2], got[3][2])
        assert g[3] == last or np.array_equal(g[1], got[3][1])


@pytest.mark.parametrize("rows,dim", [(1, 8), (5, 1000), (7, 1032), (3, 3064), (9, 4104), (6, 8192)])
@pytest.mark.parametrize("off", [0, 8])
def test_residual_layer_norm_pieces(rows, dim, off):
    """The many-row kernel at its own edges (the residual form takes it at every size): last pieces half there, one to four warps
    per row, rows 16 bytes off the widest access; against residual update and LayerNorm apart."""
    from flashrt_b200 import _lib, flash_rt_kernels as fvk
    from gpu_util import f32, rand_bf16, zeros
    rng = np.random.default_rng(rows * dim + off)
    n = rows * dim
    pad = lambda a: np.concatenate([np.zeros(off, np.uint16), a.reshape(-1)])  # noqa: E731
    x, y = pad(rand_bf16(rng, (rows, dim))), pad(rand_bf16(rng, (rows, dim)))
    g, sc, sh, w, b = (_dev(rand_bf16(rng, (dim,), 0.5)) for _ in range(5))
    s8 = f32(0.02)
    for kw, args in ((dict(scale=sc.ptr, shift=sh.ptr), (None, None, sc.ptr, sh.ptr)),
                     (dict(weight=w.ptr, bias=b.ptr), (w.ptr, b.ptr, None, None))):
        d_x, d_y, d_r, d_o = _dev(x), _dev(y), zeros((n + off,), np.uint16), zeros((n + off,), np.uint8)
        fvk.residual_layer_norm_fp8(d_x.ptr + 2 * off, d_y.ptr + 2 * off, g.ptr, d_r.ptr + 2 * off, d_o.ptr + off, s8.ptr, rows,
                                    dim, 1e-6, 0, **kw)
        d_u, d_q = _dev(x), zeros((n + off,), np.uint8)
        _lib.call("frt_b200_gate_mul_residual", d_u.ptr + 2 * off, d_y.ptr + 2 * off, g.ptr, 0, rows, dim, 0, 0)
        _lib.call("frt_b200_layer_norm", d_u.ptr + 2 * off, *args, 0, d_q.ptr + off, None, s8.ptr, rows, dim, 1e-6, 0, 0)
        assert np.array_equal(d_r.get()[off:], d_u.get()[off:]) and np.array_equal(d_o.get(), d_q.get())
