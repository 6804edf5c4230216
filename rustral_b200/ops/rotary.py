"""Rotary position embedding and SwiGLU (explicit forward / backward entry points + differentiable wrappers)."""
from __future__ import annotations

import torch

from .. import _native as N

N.optional_sig("rb_rope", [N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_int, N.c_int, N.c_int, N.c_ll, N.c_float,
                           N.c_int, N.c_void_p])
N.optional_sig("rb_swiglu_fwd", [N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_ll, N.c_int, N.c_void_p])
N.optional_sig("rb_swiglu_bwd", [N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_ll, N.c_int,
                                 N.c_void_p])


def _rope_ref(x3, pos, theta, inverse):
    T, H, D = x3.shape
    half = D // 2
    idx = torch.arange(half, dtype=torch.float32, device=x3.device)
    inv_freq = theta ** (-2.0 * idx / D)
    ang = pos.float()[:, None] * inv_freq[None, :]
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    if inverse:
        s = -s
    x0, x1 = x3[..., :half].float(), x3[..., half:].float()
    return torch.cat([x0 * c - x1 * s, x1 * c + x0 * s], -1).to(x3.dtype)


def rope_(x2: torch.Tensor, heads: int, head_dim: int, seq_len: int = 0, positions=None, pos_offset: int = 0,
          theta: float = 10000.0, inverse: bool = False) -> torch.Tensor:
    """In place on the first ``heads * head_dim`` columns of the 2-D tensor ``x2`` [tokens, >= heads*head_dim]."""
    tokens = x2.shape[0]
    if not x2.is_cuda:
        pos = positions if positions is not None else pos_offset + (torch.arange(tokens) % max(seq_len, 1))
        view = x2[:, :heads * head_dim].reshape(tokens, heads, head_dim)
        x2[:, :heads * head_dim] = _rope_ref(view, pos, theta, inverse).reshape(tokens, heads * head_dim)
        return x2
    if x2.dtype != torch.bfloat16 or x2.stride(1) != 1:
        raise TypeError("rope: bf16 rows with a contiguous last dimension are required")
    if positions is not None:
        positions = positions.to(torch.int64).contiguous()
    N.check(N.kernels().rb_rope(x2.data_ptr(), x2.stride(0), N.ptr(positions), tokens, heads, head_dim, seq_len,
                                pos_offset, theta, int(inverse), N.stream_ptr()), "rb_rope")
    return x2


N.optional_sig("rb_rope_append", [N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_int, N.c_int, N.c_int, N.c_float, N.c_void_p, N.c_void_p,
                                  N.c_void_p, N.c_ll, N.c_void_p])


def rope_append_(qkv: torch.Tensor, heads: int, kv_heads: int, head_dim: int, positions, theta: float, k_cache, v_cache, slots) -> torch.Tensor:
    """Rotates the query and key heads of qkv [tokens, (heads + 2 kv_heads) * head_dim] in place and stores keys and values in their cache
    slots (int64, negative: not stored): `rope_` and `paged.kv_append`, in one launch where that is faster."""
    shape, tokens = k_cache.shape, qkv.shape[0]
    nb, bs, hk, d = shape
    if qkv.is_cuda:
        dev, bf16 = qkv.device, torch.bfloat16
        if not (qkv.dtype is bf16 and qkv.stride(1) == 1 and hk == kv_heads and d == head_dim and v_cache.shape == shape and
                k_cache.dtype is bf16 and v_cache.dtype is bf16 and k_cache.is_contiguous() and v_cache.is_contiguous() and
                k_cache.device == dev == v_cache.device):
            raise TypeError("rope_append: bf16 rows with a contiguous last dimension and contiguous bf16 caches of the same heads are required")
        if not (slots.dtype is torch.int64 and slots.is_contiguous() and slots.dim() == 1 == positions.dim() and
                slots.shape[0] == tokens == positions.shape[0] and slots.device == dev == positions.device):
            raise TypeError("rope_append: a position and an int64 slot for every row, on its device, are required")
    # Prompts of many tokens (a thread for every lane of the GPU, see rope.cu): there the copies of the values only hold up threads that
    # rotate, and two launches are the faster way (8192 tokens, 40 heads of 128: 47.0 us against 53.3; 64 tokens: 4.6 against 3.3)
    many = tokens * ((heads + kv_heads + 3) // 4 * (head_dim // 16) + kv_heads * head_dim // 8) >= 148 * 2048
    if not qkv.is_cuda or many:
        from . import paged
        rope_(qkv, heads + kv_heads, head_dim, positions=positions, theta=theta)
        paged.kv_append(qkv[:, heads * head_dim:(heads + kv_heads) * head_dim], qkv[:, (heads + kv_heads) * head_dim:], k_cache, v_cache, slots)
        return qkv
    if positions.dtype is not torch.int64 or not positions.is_contiguous():
        positions = positions.to(torch.int64).contiguous()
    N.check(N.kernels().rb_rope_append(qkv.data_ptr(), qkv.stride(0), positions.data_ptr(), tokens, heads, kv_heads,
                                       head_dim, theta, k_cache.data_ptr(), v_cache.data_ptr(), slots.data_ptr(), nb * bs, N.stream_ptr()),
            "rb_rope_append")
    return qkv


N.optional_sig("rb_rotary_table", [N.c_void_p, N.c_void_p, N.c_float, N.c_void_p, N.c_ll, N.c_int, N.c_void_p])
N.optional_sig("rb_rotate_pairs", [N.c_void_p, N.c_ll, N.c_void_p, N.c_ll, N.c_int, N.c_ll, N.c_int, N.c_int, N.c_void_p])


def rotary_table(positions: torch.Tensor, freqs: torch.Tensor, magnitude: float = 1.0) -> torch.Tensor:
    """fp32 [rows, pairs, 2]: cosine and sine of position * freqs[pair] (fp64, on the positions' device), times `magnitude`."""
    rows, pairs = positions.numel(), freqs.numel()
    if not positions.is_cuda:
        a = positions.double()[:, None] * freqs[None, :]
        return (torch.stack([torch.cos(a), torch.sin(a)], -1) * magnitude).float()
    out = torch.empty((rows, pairs, 2), dtype=torch.float32, device=positions.device)
    if rows and pairs:
        N.check(N.kernels().rb_rotary_table(positions.data_ptr(), freqs.data_ptr(), magnitude, out.data_ptr(), rows, pairs,
                                            N.stream_ptr()), "rb_rotary_table")
    return out


def rotate_pairs(x3: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    """Reference form: a copy of x3 [rows, heads, size] with neighbouring pairs (2i, 2i + 1) of its first 2 * pairs numbers rotated."""
    y, n = x3.clone(), 2 * table.shape[1]
    c, s = table[:, None, :, 0], table[:, None, :, 1]
    u, v = x3[..., 0:n:2].float(), x3[..., 1:n:2].float()
    y[..., 0:n:2], y[..., 1:n:2] = (u * c - v * s).to(x3.dtype), (v * c + u * s).to(x3.dtype)
    return y


def rotate_halves(x3: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    """Reference form: a copy of x3 [rows, heads, size] with numbers i and i + pairs of its first 2 * pairs numbers rotated together."""
    y, n = x3.clone(), table.shape[1]
    c, s = table[:, None, :, 0], table[:, None, :, 1]
    u, v = x3[..., :n].float(), x3[..., n:2 * n].float()
    y[..., :n], y[..., n:2 * n] = (u * c - v * s).to(x3.dtype), (v * c + u * s).to(x3.dtype)
    return y


def rotate_pairs_(x2: torch.Tensor, heads: int, pitch: int, first: int, table: torch.Tensor) -> torch.Tensor:
    """In place on every head of x2 [rows, >= heads * pitch] (bf16 or fp32): the neighbouring pairs that start at column `first` of
    the head turn by `table` (see rotary_table)."""
    rows, n = x2.shape[0], 2 * table.shape[1]
    if rows == 0 or n == 0:
        return x2
    if not x2.is_cuda:
        v = x2[:, :heads * pitch].reshape(rows, heads, pitch)
        v[..., first:] = rotate_pairs(v[..., first:], table)
        x2[:, :heads * pitch] = v.reshape(rows, heads * pitch)
        return x2
    N.check(N.kernels().rb_rotate_pairs(x2[:, first:].data_ptr(), x2.stride(0), table.data_ptr(), rows, heads, pitch, table.shape[1],
                                        int(x2.dtype == torch.float32), N.stream_ptr()), "rb_rotate_pairs")
    return x2


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, seq_len, positions, pos_offset, theta):
        # x: [B, S, H, D] (contiguous); returns a rotated copy
        B, S, H, D = x.shape
        y = x.contiguous().clone().reshape(B * S, H * D)
        rope_(y, H, D, seq_len, positions, pos_offset, theta, False)
        ctx.meta = (seq_len, positions, pos_offset, theta, x.shape)
        return y.reshape(x.shape)

    @staticmethod
    def backward(ctx, dy):
        seq_len, positions, pos_offset, theta, shape = ctx.meta
        B, S, H, D = shape
        g = dy.contiguous().clone().reshape(B * S, H * D)
        rope_(g, H, D, seq_len, positions, pos_offset, theta, True)
        return g.reshape(shape), None, None, None, None


def rope(x, seq_len: int | None = None, positions=None, pos_offset: int = 0, theta: float = 10000.0):
    """Differentiable rotary embedding of [B, S, H, D]."""
    return _RopeFn.apply(x, seq_len if seq_len is not None else x.shape[1], positions, pos_offset, theta)


def swiglu_forward(gu2: torch.Tensor, out=None) -> torch.Tensor:
    tokens, F2 = gu2.shape
    F = F2 // 2
    if not gu2.is_cuda:
        g, u = gu2[:, :F].float(), gu2[:, F:].float()
        r = (g * torch.sigmoid(g) * u).to(gu2.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    out = out if out is not None else torch.empty((tokens, F), dtype=gu2.dtype, device=gu2.device)
    N.check(N.kernels().rb_swiglu_fwd(gu2.data_ptr(), gu2.stride(0), out.data_ptr(), out.stride(0), tokens, F,
                                      N.stream_ptr()), "rb_swiglu_fwd")
    return out


def swiglu_backward(dh2, gu2, out=None):
    tokens, F2 = gu2.shape
    F = F2 // 2
    if not gu2.is_cuda:
        g, u, d = gu2[:, :F].float(), gu2[:, F:].float(), dh2.float()
        s = torch.sigmoid(g)
        r = torch.cat([d * u * (s * (1 + g * (1 - s))), d * g * s], -1).to(gu2.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    out = out if out is not None else torch.empty_like(gu2)
    N.check(N.kernels().rb_swiglu_bwd(dh2.data_ptr(), dh2.stride(0), gu2.data_ptr(), gu2.stride(0), out.data_ptr(),
                                      out.stride(0), tokens, F, N.stream_ptr()), "rb_swiglu_bwd")
    return out


class _SwigluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gu):
        gu2 = gu.reshape(-1, gu.shape[-1])
        if not gu2.is_contiguous():
            gu2 = gu2.contiguous()
        ctx.save_for_backward(gu2)
        ctx.shape = gu.shape
        return swiglu_forward(gu2).reshape(*gu.shape[:-1], gu.shape[-1] // 2)

    @staticmethod
    def backward(ctx, dh):
        (gu2,) = ctx.saved_tensors
        dh2 = dh.reshape(-1, dh.shape[-1])
        if not dh2.is_contiguous():
            dh2 = dh2.contiguous()
        return swiglu_backward(dh2, gu2).reshape(ctx.shape)


def swiglu(gu):
    """``silu(gate) * up`` for ``gu = [gate | up]`` along the last dimension."""
    return _SwigluFn.apply(gu)


def swiglu_product(a: torch.Tensor, w: torch.Tensor, b_constant: bool = False) -> torch.Tensor:
    """silu(a @ gate^T) * (a @ up^T) for w = [gate; up] ([2 F, K]), for inference: one launch where the product kernels take it (bf16,
    aligned rows, up to 96 or more than 128 of them), else product and `swiglu_forward`.  The fused form does not round the two products."""
    from . import matmul
    M, K = a.shape
    F = w.shape[0] // 2
    if w.shape[0] % 2 or a.get_device() != w.get_device():
        raise ValueError("swiglu_product: as many gates as ups, on the device of the rows, are required")
    if a.is_cuda and a.dtype == w.dtype == torch.bfloat16 and M and F % 8 == 0 and K == w.shape[1] and a.stride(1) == 1 and w.stride(1) == 1 and \
            not (a.stride(0) | w.stride(0) | K) & 7 and not (a.data_ptr() | w.data_ptr()) & 15:
        out = torch.empty((M, F), dtype=a.dtype, device=a.device)
        g = N.RbGemmArgs()
        g.a, g.b, g.d = a.data_ptr(), w.data_ptr(), out.data_ptr()
        g.lda, g.ldb, g.ldd = a.stride(0), w.stride(0), F
        g.M, g.N, g.K = M, F, K
        g.act, g.alpha, g.b_constant = 9, 1.0, int(b_constant)              # RB_ACT_SWIGLU
        rc = N.kernels().rb_gemm_bf16(g, N.stream_ptr())
        if rc != -9:
            N.check(rc, "rb_gemm_bf16[swiglu]")
            return out
    return swiglu_forward(matmul.gemm(a, w, b_constant=b_constant))
