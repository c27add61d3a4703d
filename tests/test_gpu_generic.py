"""Parity of the general contraction, element-wise and aggregation kernels with the oracle."""

import ctypes

import numpy as np
import pytest
import torch

import oracle
from plaidml_b200 import kernels as K
from gpu_util import as_f32, check_close, dev, dev_bf16, empty, ptr, rng

pytestmark = pytest.mark.gpu

NP_OF = {K.F32: np.float32, K.F64: np.float64, K.I8: np.int8, K.I32: np.int32, K.I64: np.int64, K.U8: np.uint8,
         K.F16: np.float16, K.I16: np.int16, K.BOOL: np.uint8}


def run_contract(desc, srcs, out_shape, out_dtype, init=None):
    """Runs one descriptor on the GPU and through the definition-order CPU walker."""
    plan = K.Plan("contract", desc)
    d_srcs = [dev(s) for s in srcs]
    d_init = dev(init) if init is not None else None
    out = empty(out_shape, out_dtype)
    plan.contract([ptr(s) for s in d_srcs], ptr(out), ptr(d_init))
    torch.cuda.synchronize()
    ref = np.empty(out_shape, dtype=NP_OF[out_dtype])
    oracle.contract(desc, srcs, init, ref)
    return out.cpu().numpy(), ref


def gemm_desc(dt, m, n, k):
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 3, 2
    d.range[0], d.range[1], d.range[2] = m, n, k
    d.out = K.make_access(dt, [m, n], [{0: 1}, {1: 1}])
    d.src[0] = K.make_access(dt, [m, k], [{0: 1}, {2: 1}])
    d.src[1] = K.make_access(dt, [k, n], [{2: 1}, {1: 1}])
    return d


def test_contract_gemm_f32():
    g = rng(1)
    a = g.standard_normal((8, 16)).astype(np.float32)
    b = g.standard_normal((16, 32)).astype(np.float32)
    out, ref = run_contract(gemm_desc(K.F32, 8, 32, 16), [a, b], (8, 32), K.F32)
    np.testing.assert_array_equal(out, ref)  # same order of additions as the CPU walker


def test_contract_gemm_int8_wraps():
    g = rng(2)
    a = g.integers(-128, 128, size=(9, 33), dtype=np.int8)
    b = g.integers(-128, 128, size=(33, 7), dtype=np.int8)
    out, ref = run_contract(gemm_desc(K.I8, 9, 7, 33), [a, b], (9, 7), K.I8)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(out, (a.astype(np.int32) @ b.astype(np.int32)).astype(np.int8))


def test_contract_conv_with_oob_rule():
    # O[n,x,y,co] += I[n, x+i-1, y+j-1, ci] * F[i,j,ci,co]: taps outside the image are skipped
    g = rng(3)
    n, h, w, ci, co = 2, 6, 5, 3, 4
    x = g.standard_normal((n, h, w, ci)).astype(np.float32)
    f = g.standard_normal((3, 3, ci, co)).astype(np.float32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 7, 2
    for i, r in enumerate([n, h, w, co, 3, 3, ci]):
        d.range[i] = r
    d.out = K.make_access(K.F32, [n, h, w, co], [{0: 1}, {1: 1}, {2: 1}, {3: 1}])
    d.src[0] = K.make_access(K.F32, [n, h, w, ci], [{0: 1}, {1: 1, 4: 1}, {2: 1, 5: 1}, {6: 1}], offs=[0, -1, -1, 0])
    d.src[1] = K.make_access(K.F32, [3, 3, ci, co], [{4: 1}, {5: 1}, {6: 1}, {3: 1}])
    out, ref = run_contract(d, [x, f], (n, h, w, co), K.F32)
    np.testing.assert_array_equal(out, ref)
    check_close(out, oracle.conv2d_nhwc_f32(x, f, pad=(1, 1)), 1e-5)


def test_contract_maxpool_with_constraint():
    # O[x] >= I[2x + i], i < 2 as a constraint on a wider index range
    x = np.array([1, -5, 3, 9, -2, -7, 4, 0], dtype=np.float32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_MAX, K.COMBO_NONE, 2, 1
    d.range[0], d.range[1] = 4, 8
    d.out = K.make_access(K.F32, [4], [{0: 1}])
    d.src[0] = K.make_access(K.F32, [8], [{0: 2, 1: 1}])
    d.n_cons = 1
    d.cons_coef[0][1] = 1
    d.cons_range[0] = 2
    out, ref = run_contract(d, [x], (4,), K.F32)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(out, np.array([1, 9, -2, 4], dtype=np.float32))


def test_contract_non_injective_output_and_fraction():
    # O[i + j] += A[i] * B[j]  (output coordinate is not a single index) and
    # O[i] += A[i / 2] (only even i contribute)
    a = np.arange(1, 5, dtype=np.int32)
    b = np.arange(1, 4, dtype=np.int32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 2, 2
    d.range[0], d.range[1] = 4, 3
    d.out = K.make_access(K.I32, [6], [{0: 1, 1: 1}])
    d.src[0] = K.make_access(K.I32, [4], [{0: 1}])
    d.src[1] = K.make_access(K.I32, [3], [{1: 1}])
    out, ref = run_contract(d, [a, b], (6,), K.I32)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(out, np.convolve(a, b))
    d2 = K.ContractDesc()
    d2.agg, d2.combo, d2.n_idx, d2.n_src = K.AGG_SUM, K.COMBO_NONE, 1, 1
    d2.range[0] = 8
    d2.out = K.make_access(K.I32, [8], [{0: 1}])
    d2.src[0] = K.make_access(K.I32, [4], [{0: 1}], dens=[2])
    out, ref = run_contract(d2, [a], (8,), K.I32)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(out, np.array([1, 0, 2, 0, 3, 0, 4, 0], dtype=np.int32))


@pytest.mark.parametrize("seed", range(12))
def test_contract_output_dims_that_mix_variables(seed):
    # O[n, s*y + i - p, t*x - j + q, k] += I[n, y, x, c] * F[i, j, c, k] with random strides, signs, offsets and
    # an output that may be cropped: every thread solves for (y, x) from its element and walks the taps only.
    g = rng(900 + seed)
    n, h, w, c, k = (int(v) for v in g.integers(1, 5, 5))
    h, w = h + 2, w + 3
    fi, fj = int(g.integers(1, 4)), int(g.integers(1, 4))
    s, t = int(g.integers(1, 4)), int(g.integers(1, 4))
    po, qo = int(g.integers(0, 2)), int(g.integers(0, 3))
    oh = s * (h - 1) + fi - po - int(g.integers(0, 2))
    ow = t * (w - 1) + qo + 1 - int(g.integers(0, 2))
    x = g.integers(-4, 5, (n, h, w, c)).astype(np.int32)
    f = g.integers(-4, 5, (fi, fj, c, k)).astype(np.int32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 7, 2
    for i, r in enumerate([n, h, w, k, fi, fj, c]):
        d.range[i] = r
    d.out = K.make_access(K.I32, [n, oh, ow, k], [{0: 1}, {1: s, 4: 1}, {2: t, 5: -1}, {3: 1}], offs=[0, -po, qo, 0])
    d.src[0] = K.make_access(K.I32, [n, h, w, c], [{0: 1}, {1: 1}, {2: 1}, {6: 1}])
    d.src[1] = K.make_access(K.I32, [fi, fj, c, k], [{4: 1}, {5: 1}, {6: 1}, {3: 1}])
    out, ref = run_contract(d, [x, f], (n, oh, ow, k), K.I32)
    np.testing.assert_array_equal(out, ref)
    want = np.zeros((n, oh, ow, k), dtype=np.int64)
    for y in range(h):
        for xx in range(w):
            for i in range(fi):
                for j in range(fj):
                    oy, ox = s * y + i - po, t * xx - j + qo
                    if 0 <= oy < oh and 0 <= ox < ow:
                        want[:, oy, ox, :] += x[:, y, xx, :].astype(np.int64) @ f[i, j].astype(np.int64)
    np.testing.assert_array_equal(out, want.astype(np.int32))


def test_contract_shared_variable_across_output_dims():
    # O[i, i + j] = A[i, j]: the second dim's only free variable follows from the first
    a = np.arange(12, dtype=np.int32).reshape(3, 4) + 1
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_NONE, 2, 1
    d.range[0], d.range[1] = 3, 4
    d.out = K.make_access(K.I32, [3, 6], [{0: 1}, {0: 1, 1: 1}])
    d.src[0] = K.make_access(K.I32, [3, 4], [{0: 1}, {1: 1}])
    out, ref = run_contract(d, [a], (3, 6), K.I32)
    np.testing.assert_array_equal(out, ref)
    want = np.zeros((3, 6), dtype=np.int32)
    for i in range(3):
        want[i, i:i + 4] = a[i]
    np.testing.assert_array_equal(out, want)


def test_contract_init_tensor_and_min_and_cond():
    g = rng(4)
    a = g.standard_normal((5, 6)).astype(np.float32)
    bias = g.standard_normal(5).astype(np.float32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_MIN, K.COMBO_NONE, 2, 1
    d.range[0], d.range[1] = 5, 6
    d.out = K.make_access(K.F32, [5], [{0: 1}])
    d.src[0] = K.make_access(K.F32, [5, 6], [{0: 1}, {1: 1}])
    d.has_init = 1
    d.init = K.make_access(K.F32, [5], None)
    out, ref = run_contract(d, [a], (5,), K.F32, init=bias)
    np.testing.assert_array_equal(out, ref)
    np.testing.assert_array_equal(out, np.minimum(a.min(axis=1), bias))
    # cond: O[i] += (A[i] == B[i]) ? C[i] : 0
    x = np.array([1, 2, 3, 4], dtype=np.int32)
    y = np.array([1, 0, 3, 0], dtype=np.int32)
    z = np.array([10, 20, 30, 40], dtype=np.float32)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_COND, 1, 3
    d.range[0] = 4
    d.out = K.make_access(K.F32, [1], [{}])
    for s, dt in enumerate([K.I32, K.I32, K.F32]):
        d.src[s] = K.make_access(dt, [4], [{0: 1}])
    out, ref = run_contract(d, [x, y, z], (1,), K.F32)
    np.testing.assert_array_equal(out, ref)
    assert out[0] == 40.0


# --- element-wise -------------------------------------------------------------------------

def run_eltwise(op, ins, out_shape, out_dtype, in_dtypes):
    d = K.EltwiseDesc()
    d.op = op.encode()
    d.n_in, d.rank, d.out_dtype = len(ins), len(out_shape), out_dtype
    for i, s in enumerate(out_shape):
        d.sizes[i] = s
    devs = []
    for k, (a, dt) in enumerate(zip(ins, in_dtypes)):
        d.in_dtype[k] = dt
        shape = (1,) * (len(out_shape) - a.ndim) + a.shape
        stride = 1
        for i in range(len(out_shape) - 1, -1, -1):
            d.in_strides[k][i] = 0 if shape[i] == 1 and out_shape[i] != 1 else stride
            stride *= shape[i]
        devs.append(dev(a))
    plan = K.Plan("eltwise", d)
    out = empty(out_shape, out_dtype)
    plan.eltwise([ptr(t) for t in devs], ptr(out))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def test_eltwise_add_broadcast_and_relu():
    g = rng(5)
    x = g.standard_normal((4, 5, 6)).astype(np.float32)
    b = g.standard_normal(6).astype(np.float32)
    np.testing.assert_array_equal(run_eltwise("add", [x, b], (4, 5, 6), K.F32, [K.F32, K.F32]), x + b)
    np.testing.assert_array_equal(run_eltwise("relu", [x], (4, 5, 6), K.F32, [K.F32]), np.where(x < 0, 0, x))


def test_eltwise_casts_and_compare_select():
    g = rng(6)
    x = (g.standard_normal(100) * 50).astype(np.float32)
    np.testing.assert_array_equal(run_eltwise("cast", [x], (100,), K.I32, [K.F32]), x.astype(np.int32))
    i = g.integers(-1000, 1000, size=100, dtype=np.int32)
    np.testing.assert_array_equal(run_eltwise("cast", [i], (100,), K.I8, [K.I32]), i.astype(np.int8))
    np.testing.assert_array_equal(run_eltwise("cast", [i], (100,), K.F32, [K.I32]), i.astype(np.float32))
    y = g.standard_normal(100).astype(np.float32) * 50
    lt = run_eltwise("cmp_lt", [x, y], (100,), K.BOOL, [K.F32, K.F32])
    np.testing.assert_array_equal(lt, (x < y).astype(np.uint8))
    sel = run_eltwise("select", [lt, x, y], (100,), K.F32, [K.BOOL, K.F32, K.F32])
    np.testing.assert_array_equal(sel, np.where(x < y, x, y))


def test_eltwise_int_wrap_and_exp():
    a = np.array([120, -120, 5], dtype=np.int8)
    b = np.array([10, -10, 7], dtype=np.int8)
    np.testing.assert_array_equal(run_eltwise("add", [a, b], (3,), K.I8, [K.I8, K.I8]), (a + b).astype(np.int8))
    np.testing.assert_array_equal(run_eltwise("mul", [a, b], (3,), K.I8, [K.I8, K.I8]), (a * b).astype(np.int8))
    x = np.linspace(-3, 3, 64).astype(np.float32)
    np.testing.assert_allclose(run_eltwise("exp", [x], (64,), K.F32, [K.F32]), np.exp(x), rtol=1e-6)


# --- aggregation kernels ----------------------------------------------------------------------

@pytest.mark.parametrize("agg,name", [(K.AGG_MAX, "max"), (K.AGG_MIN, "min"), (K.AGG_SUM, "sum")])
@pytest.mark.parametrize("shape", [(64, 512, 1), (33, 100, 1), (8, 49, 2048), (5, 7, 3), (1, 1000, 1)])
def test_reduce_f32(agg, name, shape):
    g = rng(7)
    x = g.standard_normal(shape).astype(np.float32)
    d = K.ReduceDesc()
    d.agg, d.dtype, d.out_dtype = agg, K.F32, K.F32
    d.outer, d.reduce, d.inner = shape
    d.scale = 1.0
    plan = K.Plan("reduce", d)
    xd = dev(x)
    out = empty((shape[0], shape[2]), K.F32)
    plan.reduce(ptr(xd), ptr(out))
    torch.cuda.synchronize()
    ref = oracle.reduce_f32(x, name)
    if agg == K.AGG_SUM:
        check_close(out.cpu().numpy(), ref, 1e-5)   # order of additions differs
    else:
        np.testing.assert_array_equal(out.cpu().numpy(), ref)


def test_reduce_bf16_mean_to_f32():
    g = rng(8)
    x = dev_bf16(g.uniform(0, 1, size=(4, 49, 256)))
    d = K.ReduceDesc()
    d.agg, d.dtype, d.out_dtype = K.AGG_SUM, K.BF16, K.F32
    d.outer, d.reduce, d.inner = 4, 49, 256
    d.scale = 1.0 / 49
    plan = K.Plan("reduce", d)
    out = empty((4, 256), K.F32)
    plan.reduce(ptr(x), ptr(out))
    torch.cuda.synchronize()
    check_close(out.cpu().numpy(), oracle.reduce_f32(as_f32(x), "sum") / 49, 1e-5)


@pytest.mark.parametrize("dtype", [K.F32, K.BF16])
def test_maxpool_3x3_s2_pad1(dtype):
    g = rng(9)
    n, h, w, c = 2, 16, 16, 64
    x32 = g.standard_normal((n, h, w, c)).astype(np.float32)
    xd = dev(x32) if dtype == K.F32 else dev_bf16(x32)
    d = K.PoolDesc()
    d.agg, d.dtype = K.AGG_MAX, dtype
    d.n, d.h, d.w, d.c, d.r, d.s, d.p, d.q = n, h, w, c, 3, 3, 8, 8
    d.stride_h = d.stride_w = 2
    d.pad_h = d.pad_w = 1
    plan = K.Plan("pool", d)
    out = empty((n, 8, 8, c), dtype)
    plan.pool(ptr(xd), ptr(out))
    torch.cuda.synchronize()
    ref = oracle.pool2d_nhwc_f32(as_f32(xd), "max", (3, 3), (2, 2), (1, 1), (8, 8))
    np.testing.assert_array_equal(as_f32(out), ref)   # max is exact in any element type


def test_avgpool_excludes_padding():
    g = rng(10)
    x = g.standard_normal((1, 7, 7, 5)).astype(np.float32)
    d = K.PoolDesc()
    d.agg, d.dtype = K.AGG_SUM, K.F32
    d.n, d.h, d.w, d.c, d.r, d.s, d.p, d.q = 1, 7, 7, 5, 3, 3, 7, 7
    d.stride_h = d.stride_w = 1
    d.pad_h = d.pad_w = 1
    d.average = 1
    plan = K.Plan("pool", d)
    xd = dev(x)
    out = empty((1, 7, 7, 5), K.F32)
    plan.pool(ptr(xd), ptr(out))
    torch.cuda.synchronize()
    ref = oracle.pool2d_nhwc_f32(x, "sum", (3, 3), (1, 1), (1, 1), (7, 7), average=True)
    check_close(out.cpu().numpy(), ref, 1e-6)


def test_eltwise_dense_f32_form_gives_the_bits_of_the_general_form():
    # f32 in and out, operands dense or one value: eight elements per thread as two 16-byte pieces.  The same
    # operation on a view that is not a multiple of four elements takes the general kernel; both call one
    # arithmetic function, so the common part of their results must be equal bit for bit.
    g = rng(31)
    n = 4 * 1000 + 8
    a = g.standard_normal(n).astype(np.float32)
    b = g.uniform(0.5, 2.0, n).astype(np.float32)
    one = np.array([1.5], dtype=np.float32)
    for op_name, ins in (("add", [a, b]), ("div", [a, b]), ("max", [a, b]), ("relu", [a]), ("exp", [a]), ("tanh", [a]),
                         ("mul", [a, one]), ("sub", [one, b]), ("sqrt", [b]), ("pow", [b, a])):
        outs = []
        for count in (n, n - 3):          # dense form; general form
            arrays = [x if x.size == 1 else x[:count] for x in ins]
            strides = [[0] if x.size == 1 else [1] for x in arrays]
            d = K.EltwiseDesc()
            d.op = op_name.encode()
            d.n_in, d.rank, d.out_dtype = len(arrays), 1, K.F32
            d.sizes[0] = count
            for k, x in enumerate(arrays):
                d.in_dtype[k] = K.F32
                d.in_strides[k][0] = strides[k][0]
            plan = K.Plan("eltwise", d)
            devs = [dev(x) for x in arrays]
            out = empty((count,), K.F32)
            plan.eltwise([ptr(t) for t in devs], ptr(out))
            torch.cuda.synchronize()
            outs.append(out.cpu().numpy())
        np.testing.assert_array_equal(outs[0][:n - 3].view(np.uint32), outs[1].view(np.uint32), err_msg=op_name)
    np.testing.assert_array_equal(outs[0][:4], np.power(b[:4].astype(np.float64), a[:4].astype(np.float64)).astype(np.float32))


def test_dense_casts_between_f32_and_16_bit_floats_match_the_general_kernel():
    g = rng(32)
    n = 8 * 513
    x = (g.standard_normal(n) * 100).astype(np.float32)
    x[:6] = [np.inf, -np.inf, 0.0, -0.0, 65504.0, 1e-8]
    for narrow_dt, torch_dt in ((K.F16, torch.float16), (K.BF16, torch.bfloat16)):
        results = []
        for count in (n, n - 5):            # eight at a time; general kernel
            d = K.EltwiseDesc()
            d.op = b"cast"
            d.n_in, d.rank, d.out_dtype = 1, 1, narrow_dt
            d.sizes[0] = count
            d.in_dtype[0] = K.F32
            d.in_strides[0][0] = 1
            down = K.Plan("eltwise", d)
            src = dev(x[:count])
            half = torch.empty(count, dtype=torch_dt, device="cuda")
            down.eltwise([ptr(src)], ptr(half))
            u = K.EltwiseDesc()
            u.op = b"cast"
            u.n_in, u.rank, u.out_dtype = 1, 1, K.F32
            u.sizes[0] = count
            u.in_dtype[0] = narrow_dt
            u.in_strides[0][0] = 1
            up = K.Plan("eltwise", u)
            back = torch.empty(count, dtype=torch.float32, device="cuda")
            up.eltwise([ptr(half)], ptr(back))
            torch.cuda.synchronize()
            results.append((half.view(torch.int16).cpu().numpy(), back.cpu().numpy()))
            np.testing.assert_array_equal(back.cpu().numpy().view(np.uint32), src.to(torch_dt).to(torch.float32).cpu().numpy().view(np.uint32))
        np.testing.assert_array_equal(results[0][0][:n - 5], results[1][0])
        np.testing.assert_array_equal(results[0][1][:n - 5].view(np.uint32), results[1][1].view(np.uint32))


@pytest.mark.parametrize("dt,torch_dt", [(K.F16, torch.float16), (K.BF16, torch.bfloat16)])
def test_eltwise_dense_16_bit_form_gives_the_bits_of_the_general_form(dt, torch_dt):
    g = rng(33)
    n = 8 * 700 + 16
    a = torch.from_numpy(g.standard_normal(n).astype(np.float32)).cuda().to(torch_dt)
    b = torch.from_numpy(g.uniform(0.5, 2.0, n).astype(np.float32)).cuda().to(torch_dt)
    one = torch.tensor([1.5], device="cuda").to(torch_dt)
    for op_name, ins in (("add", [a, b]), ("mul", [a, b]), ("div", [a, b]), ("relu", [a]), ("exp", [a]), ("sub", [one, b]),
                         ("max", [a, one]), ("sqrt", [b])):
        outs = []
        for count in (n, n - 3):          # dense form; general form
            arrays = [x if x.numel() == 1 else x[:count].contiguous() for x in ins]
            d = K.EltwiseDesc()
            d.op = op_name.encode()
            d.n_in, d.rank, d.out_dtype = len(arrays), 1, dt
            d.sizes[0] = count
            for k, x in enumerate(arrays):
                d.in_dtype[k] = dt
                d.in_strides[k][0] = 0 if x.numel() == 1 else 1
            plan = K.Plan("eltwise", d)
            out = torch.empty(count, dtype=torch_dt, device="cuda")
            plan.eltwise([ptr(t) for t in arrays], ptr(out))
            torch.cuda.synchronize()
            outs.append(out.view(torch.int16).cpu().numpy())
        np.testing.assert_array_equal(outs[0][:n - 3], outs[1], err_msg=op_name)
    # and against torch for an operation whose rounding is unambiguous
    d = K.EltwiseDesc()
    d.op = b"add"
    d.n_in, d.rank, d.out_dtype = 2, 1, dt
    d.sizes[0] = n
    for k in range(2):
        d.in_dtype[k] = dt
        d.in_strides[k][0] = 1
    out = torch.empty(n, dtype=torch_dt, device="cuda")
    K.Plan("eltwise", d).eltwise([ptr(a), ptr(b)], ptr(out))
    torch.cuda.synchronize()
    assert torch.equal(out, (a.float() + b.float()).to(torch_dt))


def test_eltwise_dense_f32_with_bias_and_column_operands():
    # an operand repeated over the leading dims (a bias) or holding one value per run of the trailing dims (a column)
    # stays on the 16-byte path; +, -, *, / are correctly rounded, so numpy's float32 results are the expected bits
    from plaidml_b200.core import DType, Program
    from plaidml_b200.edsl import Placeholder
    from plaidml_b200.exec import Runner
    g = rng(34)
    cases = [((64, 256), (256,)), ((64, 256), (64, 1)), ((4, 8, 16), (8, 16)), ((4, 8, 16), (4, 8, 1)), ((4, 8, 16), (4, 1, 16)),
             ((6, 20), (20,)), ((5, 8), (5, 1))]
    for big, small in cases:
        x = g.standard_normal(big).astype(np.float32)
        y = g.uniform(0.5, 2.0, small).astype(np.float32)
        X, Y = Placeholder(DType.FLOAT32, list(big)), Placeholder(DType.FLOAT32, list(small))
        outs = Runner(Program("bcast", [X, Y], [X + Y, X * Y, Y - X, X / Y]), "cuda.0").run([x, y])
        for got, want in zip(outs, (x + y, x * y, y - x, x / y)):
            np.testing.assert_array_equal(got.view(np.uint32), want.astype(np.float32).view(np.uint32), err_msg=f"{big} {small}")


# --- the strided form (lean kernels) and matrix products of the general contraction -----------------------------------

def strided_case(seed):
    """A windowed contraction with strides, dilation, padding, mirrored taps, a constraint or an initial value now and
    then; every aggregation and combination, depthwise or with its own output channels."""
    g = rng(7000 + seed)
    pick = lambda *xs: xs[int(g.integers(0, len(xs)))]
    dt = pick(K.F32, K.F32, K.F64, K.I32, K.I8)
    n, h, w, c, co = 1 + int(g.integers(0, 2)), *(int(v) for v in g.integers(3, 9, 2)), pick(1, 3, 4, 5, 8), pick(1, 4, 6)
    r, s, p, q = (int(v) for v in (*g.integers(1, 4, 2), *g.integers(1, 8, 2)))
    st, dl, pd = g.integers(1, 3, 2), g.integers(1, 3, 2), g.integers(-1, 3, 2)
    mirror = seed % 2
    d = K.ContractDesc()
    d.agg = pick(K.AGG_SUM, K.AGG_SUM, K.AGG_MAX, K.AGG_MIN, K.AGG_PROD, K.AGG_ASSIGN)
    d.combo = pick(K.COMBO_MUL, K.COMBO_MUL, K.COMBO_ADD, K.COMBO_NONE)
    d.n_src = 1 if d.combo == K.COMBO_NONE else 2
    N, Y, X, C, I, J, CI = range(7)
    depthwise = seed % 3 != 0
    ranges = [n, p, q, c, r, s] if depthwise else [n, p, q, co, r, s, c]
    d.n_idx = len(ranges)
    for i, v in enumerate(ranges):
        d.range[i] = v
    shape = (n, p, q, ranges[3])
    d.out = K.make_access(dt, shape, [{N: 1}, {Y: 1}, {X: 1}, {C: 1}])
    rows = {Y: int(st[0]), I: int(-dl[0] if mirror else dl[0])}
    d.src[0] = K.make_access(dt, [n, h, w, c], [{N: 1}, rows, {X: int(st[1]), J: int(dl[1])}, {C if depthwise else CI: 1}],
                             offs=[0, int(-pd[0] + mirror * dl[0] * (r - 1)), int(-pd[1]), 0])
    taps = (r, s, c) if depthwise else (r, s, c, co)
    d.src[1] = K.make_access(dt, taps, [{I: 1}, {J: 1}, {C: 1}] if depthwise else [{I: 1}, {J: 1}, {CI: 1}, {C: 1}])
    if seed % 4 == 0:
        d.n_cons, d.cons_coef[0][I], d.cons_coef[0][X], d.cons_off[0], d.cons_range[0] = 1, 1, 1, -1, 4
    draw = lambda sh: (g.standard_normal(sh) * (40 if dt == K.I8 else 3)).astype(NP_OF[dt])
    init = None
    if seed % 5 == 0:
        d.has_init, init = 1, draw(shape[-1:])
        d.init = K.make_access(dt, shape, None, strides=[0, 0, 0, 1])
    return d, [draw((n, h, w, c)), draw(taps)][:d.n_src], shape, dt, init


@pytest.mark.parametrize("seed", range(48))
def test_strided_contraction_equals_the_walker(seed):
    d, srcs, shape, dt, init = strided_case(seed)
    out, ref = run_contract(d, srcs, shape, dt, init)
    np.testing.assert_array_equal(out, ref)   # same terms, same order, every operation rounded on its own


@pytest.mark.parametrize("n,hw,c,r,stride,dil,pad,per_channel,swap", [
    (23, 33, 52, 3, 1, 1, 1, True, False),      # quads; runs end inside a row (33 = 8 * 4 + 1)
    (23, 33, 51, 3, 1, 1, 1, True, True),       # single elements, filter as the first operand
    (60, 40, 56, 3, 2, 1, 1, True, False),      # neighbours two columns apart: no shared elements
    (33, 30, 48, 2, 1, 2, 0, True, False),      # dilation 2 against stride 1
    (75, 31, 64, 4, 2, 2, 3, True, False),      # stride equal to the dilation, padding beyond the first tap
    (23, 33, 52, 3, 1, 1, 1, False, False),     # one filter for all channels
])
def test_runs_of_neighbours_in_one_thread(n, hw, c, r, stride, dil, pad, per_channel, swap):
    g = rng(7100 + hw + c)
    p = (hw + 2 * pad - dil * (r - 1) - 1) // stride + 1
    N, Y, X, C, I, J = range(6)
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 6, 2
    for i, v in enumerate([n, p, p, c, r, r]):
        d.range[i] = v
    assert n * p * -(-p // 4) * (c // 4 if c % 4 == 0 else c) >= 75776   # wide enough for the kernel in question
    d.out = K.make_access(K.F32, [n, p, p, c], [{N: 1}, {Y: 1}, {X: 1}, {C: 1}])
    x_acc = K.make_access(K.F32, [n, hw, hw, c], [{N: 1}, {Y: stride, I: dil}, {X: stride, J: dil}, {C: 1}], offs=[0, -pad, -pad, 0])
    f_shape = (r, r, c) if per_channel else (r, r)
    f_acc = K.make_access(K.F32, f_shape, [{I: 1}, {J: 1}, {C: 1}][:len(f_shape)])
    x, f = g.standard_normal((n, hw, hw, c)).astype(np.float32), g.standard_normal(f_shape).astype(np.float32)
    d.src[0], d.src[1] = (f_acc, x_acc) if swap else (x_acc, f_acc)
    out, ref = run_contract(d, [f, x] if swap else [x, f], (n, p, p, c), K.F32)
    # r * r terms added in the same order, one rounding per term here and two in the walker: each at most 2^-24 of a
    # partial sum, which stays below the sum of the terms' magnitudes
    bound = 3 * r * r * 2.0 ** -24 * np.abs(f).max() * np.abs(x).max() * r * r
    assert np.max(np.abs(out - ref)) <= bound


@pytest.mark.parametrize("seed", range(24))
def test_products_in_any_order_of_dims(seed):
    # every order of the dims of both operands and of the result: transposed operands, batch dims outside or inside,
    # orders that no single matrix product covers (these stay with the strided form)
    g = rng(7200 + seed)
    ext = {"m": int(g.integers(1, 150)), "n": int(g.integers(1, 150)), "k": int(g.integers(1, 300)), "b": int(g.integers(1, 4))}
    while ext["m"] * ext["n"] * ext["k"] * ext["b"] <= 32768:
        ext["k"] = 2 * ext["k"] + 1
    var = {v: i for i, v in enumerate("mnkb")}
    a, b, c = ("".join(g.permutation(list(v))) for v in ("mkb", "knb", "mnb"))
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 4, 2
    for v, i in var.items():
        d.range[i] = ext[v]
    acc = lambda dims: K.make_access(K.F32, [ext[v] for v in dims], [{var[v]: 1} for v in dims])
    d.out, d.src[0], d.src[1] = acc(c), acc(a), acc(b)
    x, y = (g.standard_normal([ext[v] for v in dims]).astype(np.float32) for dims in (a, b))
    out, ref = run_contract(d, [x, y], tuple(ext[v] for v in c), K.F32)
    want = np.einsum(f"{a},{b}->{c}", x.astype(np.float64), y.astype(np.float64))
    norm = np.linalg.norm(want)
    # no further from the exact sums than the one-by-one f32 sums, or than 2^-20 where there are few terms
    assert np.linalg.norm(out - want) / norm <= max(1.5 * np.linalg.norm(ref - want) / norm, 2.0 ** -20)


@pytest.mark.parametrize("a,b,c,ext", [
    ("ij", "ij", "ij", {"i": 211, "j": 307}),                # all batch dims
    ("yc", "c", "yc", {"y": 25089, "c": 24}),                # a scale per channel
    ("ij", "i", "ij", {"i": 130, "j": 1001}),
    ("i", "j", "ij", {"i": 513, "j": 770}),                  # no terms
    ("km", "kn", "mn", {"m": 130, "n": 70, "k": 15}),        # too few terms
    ("ik", "ik", "i", {"i": 5000, "k": 40}),                 # one dot product per batch entry
    ("bkm", "bkn", "bmn", {"b": 3000, "m": 4, "n": 3, "k": 20}),
])
def test_products_that_leave_their_tiles_empty_add_term_by_term(a, b, c, ext):
    g = rng(7250 + len(ext))
    var = {v: i for i, v in enumerate(ext)}
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, len(ext), 2
    for v, i in var.items():
        d.range[i] = ext[v]
    acc = lambda dims: K.make_access(K.F32, [ext[v] for v in dims], [{var[v]: 1} for v in dims])
    d.out, d.src[0], d.src[1] = acc(c), acc(a), acc(b)
    x, y = (g.standard_normal([ext[v] for v in dims]).astype(np.float32) for dims in (a, b))
    out, ref = run_contract(d, [x, y], tuple(ext[v] for v in c), K.F32)
    np.testing.assert_array_equal(out, ref)


def test_more_products_than_a_launch_takes_tiles():
    n = (1 << 28) + 3
    x, y = (torch.rand(n, device="cuda") - 0.5 for _ in range(2))
    out = torch.empty(n, device="cuda")
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 1, 2
    d.range[0] = n
    d.out = K.make_access(K.F32, [n], [{0: 1}])
    d.src[0] = d.src[1] = K.make_access(K.F32, [n], [{0: 1}])
    K.Plan("contract", d).contract([ptr(x), ptr(y)], ptr(out))
    assert torch.equal(out, x * y)


@pytest.mark.parametrize("a,b,c,m,n,k", [("km", "kn", "mn", 130, 70, 64), ("km", "kn", "mn", 40, 36, 2000), ("mk", "nk", "nm", 150, 40, 48),
                                         ("km", "nk", "mn", 129, 131, 130), ("mk", "kn", "mn", 300, 200, 515)])
def test_products_of_infinite_and_of_tiny_operands(a, b, c, m, n, k):
    ext = {"m": m, "n": n, "k": k}
    var = {v: i for i, v in enumerate(ext)}
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 3, 2
    for v, i in var.items():
        d.range[i] = ext[v]
    acc = lambda dims: K.make_access(K.F32, [ext[v] for v in dims], [{var[v]: 1} for v in dims])
    d.out, d.src[0], d.src[1] = acc(c), acc(a), acc(b)
    g = rng(7400 + k)
    x, y = g.uniform(0.5, 1, (m, k)).astype(np.float32), g.uniform(0.5, 1, (k, n)).astype(np.float32)
    x[3, 5], x[7, k - 1], x[9, 2] = np.inf, -np.inf, np.nan
    y[5, 4], y[5, 6], y[k - 1, 8] = 2.0 ** -140, 0.0, -(2.0 ** -149)     # inf times these: inf, NaN, +inf
    x[11] *= 2.0 ** -120                                                  # rows whose parts would end above their last bits
    x[13] *= 2.0 ** -130
    x[15] = 0
    out, _ = run_contract(d, [np.ascontiguousarray(v) for v in (x if a == "mk" else x.T, y if b == "kn" else y.T)], tuple(ext[v] for v in c), K.F32)
    got = out if c == "mn" else out.T
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ y.astype(np.float64)
        off = np.abs(got - want)
    np.testing.assert_array_equal(np.where(np.isfinite(got), 0, got), np.where(np.isfinite(want), 0, want))
    fine = np.isfinite(want)
    # plain f32 sums: k roundings of at most 2^-24 of a sum of positive terms, and 2^-150 where a term is subnormal
    assert np.all(off[fine] <= k * (2.0 ** -24 * np.abs(want[fine]) + 2.0 ** -150))


def test_contractions_add_term_by_term_without_k_split(monkeypatch):
    # a matrix product and a depthwise filter, both large enough for kernels with other roundings
    monkeypatch.setenv("PMLB_SPLIT_K", "0")
    g = rng(7500)
    m, n, k = 90, 70, 33
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 3, 2
    for i, v in enumerate([m, n, k]):
        d.range[i] = v
    d.out = K.make_access(K.F32, [m, n], [{0: 1}, {1: 1}])
    d.src[0] = K.make_access(K.F32, [k, m], [{2: 1}, {0: 1}])
    d.src[1] = K.make_access(K.F32, [k, n], [{2: 1}, {1: 1}])
    out, ref = run_contract(d, [g.standard_normal(s).astype(np.float32) for s in ((k, m), (k, n))], (m, n), K.F32)
    np.testing.assert_array_equal(out, ref)
    rows, c, r = 20000, 51, 3      # 5000 runs of 51: wide enough for runs of neighbours
    d = K.ContractDesc()
    d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 3, 2
    for i, v in enumerate([rows, c, r]):
        d.range[i] = v
    d.out = K.make_access(K.F32, [rows, c], [{0: 1}, {1: 1}])
    d.src[0] = K.make_access(K.F32, [rows + r - 1, c], [{0: 1, 2: 1}, {1: 1}])
    d.src[1] = K.make_access(K.F32, [r, c], [{2: 1}, {1: 1}])
    out, ref = run_contract(d, [g.standard_normal(s).astype(np.float32) for s in ((rows + r - 1, c), (r, c))], (rows, c), K.F32)
    np.testing.assert_array_equal(out, ref)


def test_contraction_plans_are_made_and_freed_while_a_stream_is_captured():
    # a matrix product and a strided contraction; the graph outlives the plans
    m, n, k = 160, 96, 700
    x, y = torch.randn(k, m, device="cuda"), torch.randn(k, n, device="cuda")
    s = torch.randn(n, device="cuda")
    out, scaled = torch.zeros(m, n, device="cuda"), torch.zeros(m, n, device="cuda")

    def desc(src_b, b, n_idx):
        d = K.ContractDesc()
        d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, n_idx, 2
        for i, v in enumerate([m, n, k][:n_idx]):
            d.range[i] = v
        d.out = K.make_access(K.F32, [m, n], [{0: 1}, {1: 1}])
        d.src[0] = K.make_access(K.F32, [k, m], [{2: 1}, {0: 1}]) if n_idx == 3 else d.out
        d.src[1] = K.make_access(K.F32, src_b, b)
        return d

    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        product = K.Plan("contract", desc([k, n], [{2: 1}, {1: 1}], 3))
        product.contract([ptr(x), ptr(y)], ptr(out), stream=stream.cuda_stream)
        scale = K.Plan("contract", desc([n], [{1: 1}], 2))
        scale.contract([ptr(out), ptr(s)], ptr(scaled), stream=stream.cuda_stream)
        del product, scale
    for _ in range(2):
        x.normal_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = x.double().t() @ y.double()
        assert torch.linalg.norm(out.double() - want) <= 1e-6 * torch.linalg.norm(want)
        assert torch.equal(scaled, out * s)


def test_product_that_does_not_cover_its_output_or_reads_out_of_range_stays_exact():
    # a range shorter than the output dim leaves the identity there; one longer than an operand's dim skips terms
    g = rng(7300)
    a, b = g.standard_normal((64, 50)).astype(np.float32), g.standard_normal((64, 60)).astype(np.float32)
    for m, k, rows in ((40, 64, 50), (50, 70, 50)):
        d = K.ContractDesc()
        d.agg, d.combo, d.n_idx, d.n_src = K.AGG_SUM, K.COMBO_MUL, 3, 2
        for i, v in enumerate([m, 60, k]):
            d.range[i] = v
        d.out = K.make_access(K.F32, [rows, 60], [{0: 1}, {1: 1}])
        d.src[0] = K.make_access(K.F32, [64, 50], [{2: 1}, {0: 1}])
        d.src[1] = K.make_access(K.F32, [64, 60], [{2: 1}, {1: 1}])
        out, ref = run_contract(d, [a, b], (rows, 60), K.F32)
        np.testing.assert_array_equal(out, ref)


@pytest.mark.parametrize("graph", [False, True], ids=["stream", "graph"])
def test_a_chain_of_short_launches_reads_what_the_launch_before_wrote(graph):
    # launches may begin before their predecessor has ended: two buffers written in turn by element-wise steps and by
    # products with a permutation (exact), 200 launches
    rows, n = 256, 128
    perm = torch.eye(n, device="cuda")[torch.arange(n).roll(1)].contiguous()
    one = torch.ones(1, device="cuda")
    x0 = torch.randint(0, 1000, (rows, n), device="cuda").float()

    e = K.EltwiseDesc()
    e.op, e.n_in, e.rank, e.out_dtype = b"add", 2, 2, K.F32
    e.in_dtype[0] = e.in_dtype[1] = K.F32
    e.sizes[0], e.sizes[1] = rows, n
    e.in_strides[0][0], e.in_strides[0][1] = n, 1
    add = K.Plan("eltwise", e)
    d = K.GemmDesc()
    d.in_dtype = d.out_dtype = K.F32
    d.m, d.n, d.k, d.batch = rows, n, n, 1
    d.lda, d.ldb, d.ldc = n, n, n
    mul = K.Plan("gemm", d)

    x, y = x0.clone(), torch.empty_like(x0)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())

    def chain():
        for _ in range(50):
            add.eltwise([ptr(x), ptr(one)], ptr(y), stream=stream.cuda_stream)
            mul.gemm(ptr(y), ptr(perm), ptr(x), stream=stream.cuda_stream)
            add.eltwise([ptr(x), ptr(one)], ptr(y), stream=stream.cuda_stream)
            add.eltwise([ptr(y), ptr(one)], ptr(x), stream=stream.cuda_stream)

    with torch.cuda.stream(stream):
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                chain()
            g.replay()
        else:
            chain()
    stream.synchronize()
    got = x.cpu()
    moved = x0.cpu().numpy() @ np.linalg.matrix_power(perm.cpu().numpy(), 50) + 150
    np.testing.assert_array_equal(got.numpy(), moved.astype(np.float32))
