"""Gather kernels and the differentiable ops: the five check families of the reference's unit test
(modal/test_moe_permute.py:50-91), same shapes (n=64, d=256, E=16, k in {6,12}, f32 and bf16) and
tolerances (0 for plain gathers, 1e-5 f32, 2e-2 bf16)."""
import numpy as np
import pytest
import torch

import oracle as O
from util import rand_routing, softmax_np, to_dev, to_np

pytestmark = pytest.mark.gpu
E = 16


def prep(a, dtype):
  return O.bf16_round(a) if dtype == torch.bfloat16 else a.astype(np.float32)


@pytest.mark.parametrize("dtype,k", [(torch.float32, 6), (torch.bfloat16, 6), (torch.bfloat16, 12), (torch.float32, 12)])
@pytest.mark.parametrize("n,d", [(64, 256), (60, 256), (64, 1024), (33, 2048), (16, 8)])
def test_reference_check_families(cuda, dtype, k, n, d):
  from lewi_surge_b200 import ops
  tol = 2e-2 if dtype == torch.bfloat16 else 1e-5
  rng = np.random.default_rng(k * 7 + (dtype == torch.bfloat16) + n + d)
  x = prep(rng.standard_normal((n, d)), dtype)
  flat = rand_routing(rng, n, E, k).reshape(-1)
  w = softmax_np(rng.standard_normal((n, k)).astype(np.float32))
  m = n * k
  y = prep(rng.standard_normal((m, d)), dtype)
  g = prep(rng.standard_normal((n, d)), dtype)
  order, pos = O.sort_indices(flat, E)
  pos2 = pos.reshape(n, k)
  idx = (rng.permutation(m) % n).astype(np.int32)
  scale = rng.standard_normal(m).astype(np.float32)
  X, Y, G = (to_dev(a, dtype, cuda) for a in (x, y, g))
  I, P, W, S = to_dev(idx, torch.int32, cuda), to_dev(pos2, torch.int32, cuda), to_dev(w, torch.float32, cuda), to_dev(scale, torch.float32, cuda)

  # 1. kernels vs references
  assert np.array_equal(to_np(ops.gather_rows(X, I)), x[idx])                      # exact (tol 0)
  want = O.gather_rows(x, idx, scale, out_bf16=dtype == torch.bfloat16)
  assert O.rel_err(to_np(ops.gather_rows(X, I, S)), want) <= (0 if dtype == torch.float32 else tol)
  assert O.rel_err(to_np(ops.gather_reduce(Y, P, None, torch.float32)), O.gather_reduce(y, pos2)) <= tol
  assert O.rel_err(to_np(ops.gather_reduce(Y, P, W, torch.float32)), O.gather_reduce(y, pos2, w)) <= tol
  assert O.rel_err(to_np(ops.gather_reduce(Y, P, W)), O.gather_reduce(y, pos2, w)) <= tol   # input dtype out
  assert O.rel_err(to_np(ops.gather_dot(Y, P, G)), O.gather_dot(y, pos2, g)) <= tol

  # 2. sort_indices
  o2, p2 = ops.sort_indices(to_dev(flat, torch.int32, cuda), E)
  assert np.array_equal(to_np(o2), order) and np.array_equal(to_np(p2), pos)

  # 3. dispatch -> tanh expert -> combine, forward and gradients
  ops.CFG["num_experts"] = E
  Xg = X.clone().requires_grad_(True)
  Wg = W.clone().requires_grad_(True)
  out = ops.moe_block(Xg, to_dev(flat, torch.int32, cuda), Wg, lambda r: torch.tanh(r.float()).to(r.dtype))
  loss = (out * G.float()).sum()
  loss.backward()
  xs = O.dispatch(x, order, pos)
  ye = prep(np.tanh(xs), dtype)
  ref_out = O.combine(ye, order, pos, w)
  assert O.rel_err(to_np(out), ref_out) <= tol
  assert O.rel_err(loss.item(), float((ref_out * g).sum())) <= tol
  dy, dw = O.combine_bwd(g, ye, order, pos, w)
  dx = O.dispatch_bwd(dy * (1 - np.tanh(xs) ** 2), order, pos, n)
  assert O.rel_err(to_np(Xg.grad), dx) <= tol
  assert O.rel_err(to_np(Wg.grad), dw) <= tol

  # 4. permute_rows gradient
  perm = rng.permutation(m).astype(np.int32)
  Yg = Y.clone().requires_grad_(True)
  gi = to_dev(x[idx], dtype, cuda)
  (ops.permute_rows(Yg, to_dev(perm, torch.int32, cuda)).float() * gi.float()).sum().backward()
  assert O.rel_err(to_np(Yg.grad), O.permute_rows_bwd(x[idx], perm)) <= tol


def test_gather_edge_cases(cuda):
  from lewi_surge_b200 import ops, _lib
  x = torch.randn(8, 64, device=cuda).to(torch.bfloat16)
  # negative index -> zero row; empty index list -> empty output
  out = ops.gather_rows(x, torch.tensor([3, -1, 0], dtype=torch.int32, device=cuda))
  assert torch.equal(out[0], x[3]) and torch.equal(out[2], x[0]) and bool((out[1] == 0).all())
  assert ops.gather_rows(x, torch.zeros(0, dtype=torch.int32, device=cuda)).shape == (0, 64)
  # out-of-range index is skipped and reported, never dereferenced
  _lib.last_status()
  ops.gather_rows(x, torch.tensor([100], dtype=torch.int32, device=cuda))
  assert _lib.last_status() & _lib.STATUS_BAD_INDEX
  # unsupported row size raises (no fallback)
  with pytest.raises(_lib.LewiError):
    ops.gather_rows(torch.zeros(4, 7, device=cuda), torch.zeros(2, dtype=torch.int32, device=cuda))


def test_gather_reduce_addends_and_padded_rows(cuda):
  from lewi_surge_b200 import ops
  rng = np.random.default_rng(0)
  n, k, d = 50, 6, 512
  y = O.bf16_round(rng.standard_normal((n * k + 100, d)))
  pos = rng.permutation(n * k + 100)[: n * k].reshape(n, k).astype(np.int32)
  w = softmax_np(rng.standard_normal((n, k)).astype(np.float32))
  a0 = O.bf16_round(rng.standard_normal((n, d)))
  a1 = O.bf16_round(rng.standard_normal((n, d)))
  got = ops.gather_reduce(to_dev(y, torch.bfloat16, cuda), to_dev(pos, torch.int32, cuda), to_dev(w, torch.float32, cuda),
                          torch.float32, add0=to_dev(a0, torch.bfloat16, cuda), add1=to_dev(a1, torch.bfloat16, cuda))
  assert O.rel_err(to_np(got), O.gather_reduce(y, pos, w) + a0 + a1) <= 1e-5


def test_full_size_dispatch_combine_round_trip(cuda):
  """Config-2 size: dispatch then unweighted combine of the same rows gives k * x exactly (bf16 integers)."""
  from lewi_surge_b200 import ops, layer
  t, e, k, d = 32768, 128, 6, 1024
  g = torch.Generator(device="cpu").manual_seed(0)
  x = torch.randint(-8, 9, (t, d), generator=g).to(torch.bfloat16).to(cuda)
  logits = torch.randn((t, e), generator=g).to(cuda)
  tb = layer.router_topk(logits, k)
  xs = ops.dispatch(x, tb.order, tb.pos)
  assert torch.equal(xs, x[(tb.order // k).long()])
  back = ops.gather_reduce(xs, tb.pos.view(t, k), None, torch.float32)
  assert torch.equal(back, x.float() * k)


@pytest.mark.parametrize("t,e,k,d,skew", [(300, 8, 2, 128, False), (4096, 64, 6, 1024, False), (5000, 128, 6, 256, True),
                                          (30000, 16, 6, 136, False)])
def test_dispatch_rows_equals_the_row_gather(cuda, t, e, k, d, skew):
  """The token-order dispatch writes exactly what the gather through row_slot writes, zero padding rows included."""
  from lewi_surge_b200 import layer, ops, _lib
  g = torch.Generator(device="cpu").manual_seed(t + k)
  logits = torch.randn((t, e), generator=g) * 2
  if skew:
    logits = logits + torch.from_numpy(O.zipf_bias(e, 0))
  tb = layer.router_topk(logits.to(cuda), k)
  x = torch.randn((t, d), generator=g).to(torch.bfloat16).to(cuda)
  _lib.last_status()
  want = torch.full((tb.mpad, d), 7.0, dtype=torch.bfloat16, device=cuda)
  got = want.clone()
  ops.gather_rows(x, tb.row_slot, idx_div=k, out=want, n_rows_dev=tb.n_blocks, rows_per_unit=128)
  ops.dispatch_rows(x, tb.pad_pos.view(t, k), tb.row_slot, out=got, n_rows_dev=tb.n_blocks, rows_per_unit=128)
  assert _lib.last_status() == 0
  assert torch.equal(got, want)           # rows past the live blocks keep the fill value in both
  nb = int(tb.n_blocks.item()) * 128
  assert bool((got[nb:] == 7).all()) and nb <= tb.mpad


@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                       (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("k", [1, 8, 9, 32])
def test_gather_reduce_of_few_rows_gives_the_bits_of_many(cuda, dtype, out, k):
  """Few rows (how many depends on k and d: here up to 132 at k = 1 and 2300 at k >= 8) take another kernel than many: 1, 3 and 700
  rows against the same rows of a call of 10000, with weights, both addends, absent rows and a row length that fills no warp."""
  from lewi_surge_b200 import ops
  d, n, m = 264, 10000, 500
  gen = torch.Generator(device=cuda).manual_seed(k)
  y, a0, a1 = (torch.randn(r, d, generator=gen, device=cuda).to(dtype) for r in (m, n, n))
  pos = torch.randint(-1, m, (n, k), generator=gen, device=cuda, dtype=torch.int32)
  w = torch.rand(n, k, generator=gen, device=cuda)
  many = ops.gather_reduce(y, pos, w, out, add0=a0, add1=a1)
  bare = ops.gather_reduce(y, pos, None, out)
  for r in (1, 3, 700):
    assert torch.equal(ops.gather_reduce(y, pos[:r], w[:r], out, add0=a0[:r], add1=a1[:r]), many[:r])
    assert torch.equal(ops.gather_reduce(y, pos[:r], None, out), bare[:r])


@pytest.mark.parametrize("t,k,d,dtype,g_dtype", [(1, 1, 8, "bf16", "f32"), (3, 32, 4, "f32", "f32"), (33, 7, 264, "bf16", "bf16"),
                                                 (700, 6, 1032, "bf16", "f32"), (129, 12, 1028, "f32", "f32"), (70, 6, 2048, "f32", "f32"), (60, 6, 4096, "bf16", "f32"),
                                                 (2500, 3, 256, "f32", "f32")])
def test_token_order_dispatch_and_combine_gradients_equal_the_row_gathers(cuda, t, k, d, dtype, g_dtype):
  """Same bits as gather_rows / scaled gather_rows / gather_dot on the inverse permutation, through the public functions' gradients too."""
  from lewi_surge_b200 import ops, _lib
  dt = dict(bf16=torch.bfloat16, f32=torch.float32)
  gen = torch.Generator(device=cuda).manual_seed(t + k)
  order = torch.randperm(t * k, generator=gen, device=cuda).to(torch.int32)
  pos = torch.empty_like(order)
  pos[order.long()] = torch.arange(t * k, dtype=torch.int32, device=cuda)
  rnd = lambda *s: torch.randn(*s, generator=gen, device=cuda)
  x, y, w, g = rnd(t, d).to(dt[dtype]), rnd(t * k, d).to(dt[dtype]), rnd(t, k), rnd(t, d).to(dt[g_dtype])
  _lib.last_status()
  assert torch.equal(ops.dispatch(x, order, pos), ops.gather_rows(x, order, idx_div=k))
  gy = g.to(y.dtype)
  dy, dw = ops.combine_bwd(y, pos.view(t, k), g, w)
  assert torch.equal(dy, ops.gather_rows(gy, order, w.reshape(-1), idx_div=k, scale_by_idx=True))
  assert torch.equal(dw, ops.gather_dot(y, pos.view(t, k), gy))
  y.requires_grad_(True)
  w.requires_grad_(True)
  got = torch.autograd.grad(ops.combine(y, order, pos, w), (y, w), g.float())
  assert torch.equal(got[0], dy) and torch.equal(got[1], dw)
  assert _lib.last_status() == 0


@pytest.mark.parametrize("t,k,d,dtype", [(1, 2, 8, "bf16"), (50, 6, 264, "f32"), (700, 4, 1024, "bf16"), (40, 12, 2048, "f32"), (6000, 3, 64, "bf16"),
                                       (1479, 2, 264, "f32"), (1480, 32, 264, "f32"), (2000, 6, 1032, "bf16")])
@pytest.mark.parametrize("tables", ["dropped", "order_only", "pos_only", "unrelated", "short"])
def test_dispatch_and_combine_with_tables_that_are_no_permutations(cuda, t, k, d, dtype, tables):
  """Slots that were dropped (both tables negative, or one of them), tables that do not belong together, rows left out of order: every row is
  what the row gathers make of `order`, every sum and dot what `pos` names, and nothing is left unwritten."""
  from lewi_surge_b200 import ops, _lib
  dt = dict(bf16=torch.bfloat16, f32=torch.float32)[dtype]
  gen = torch.Generator(device=cuda).manual_seed(t + k)
  rnd = lambda *s: torch.randn(*s, generator=gen, device=cuda)
  m = t * k
  order = torch.randperm(m, generator=gen, device=cuda).to(torch.int32)
  pos = torch.empty_like(order)
  pos[order.long()] = torch.arange(m, dtype=torch.int32, device=cuda)
  gone = torch.rand(m, generator=gen, device=cuda) < 0.3
  gone[0] = True
  rows = m
  if tables in ("dropped", "pos_only"):
    pos[order[gone].long()] = -1
  if tables in ("dropped", "order_only"):
    order[gone] = -1
  if tables == "unrelated":   # some rows name the same slot, some slots the same row, out of range of nothing
    order = torch.randint(-1, m, (m,), generator=gen, device=cuda, dtype=torch.int32)
    pos = torch.randint(-1, m, (m,), generator=gen, device=cuda, dtype=torch.int32)
  if tables == "short":       # the dropped slots' rows do not exist at all
    rows = m // 2 + 1
    order = order[:rows].contiguous()
    pos = torch.where(pos < rows, pos, -1)
  x, y, w, g = rnd(t, d).to(dt), rnd(rows, d).to(dt), rnd(t, k), rnd(t, d)
  junk = torch.full((4 * m * d,), float("nan"), device=cuda)
  del junk                    # what a fresh output may hold
  _lib.last_status()
  x.requires_grad_(True)
  if tables != "short":       # (k of the dispatch follows from the rows)
    out = ops.dispatch(x, order, pos)
    assert torch.equal(out, ops.gather_rows(x, order, idx_div=k))
    dx, = torch.autograd.grad(out, x, y)
    assert torch.equal(dx, ops.gather_reduce(y, pos.view(t, k), None, dt))
  y.requires_grad_(True)
  w.requires_grad_(True)
  dy, dw = torch.autograd.grad(ops.combine(y, order, pos, w), (y, w), g)
  gy = g.to(dt)
  assert torch.equal(dy, ops.gather_rows(gy, order, w.detach().reshape(-1), idx_div=k, scale_by_idx=True))
  assert torch.equal(dw, ops.gather_dot(y.detach(), pos.view(t, k), gy))
  assert _lib.last_status() == 0


def test_a_slot_without_a_row_is_an_error_where_pos_alone_is_given(cuda):
  from lewi_surge_b200 import ops, _lib
  x, pos = torch.randn(2, 64, device=cuda), torch.tensor([0, 3, -1, 1], dtype=torch.int32, device=cuda)
  _lib.last_status()
  ops.dispatch_tokens(x, pos, 2)
  assert _lib.last_status() & _lib.STATUS_BAD_INDEX
  ops.combine_bwd(torch.randn(4, 64, device=cuda), pos.view(2, 2), x, torch.rand(2, 2, device=cuda))
  assert _lib.last_status() & _lib.STATUS_BAD_INDEX
  order = torch.tensor([0, 3, 4, 1], dtype=torch.int32, device=cuda)   # slot 4 of four: skipped and reported, as by gather_rows
  ops.dispatch(x, order, pos)
  assert _lib.last_status() & _lib.STATUS_BAD_INDEX


@pytest.mark.parametrize("dtype,g_dtype", [("bf16", "f32"), ("bf16", "f16"), ("f32", "bf16")])
def test_combine_gradients_take_an_upstream_gradient_at_any_address(cuda, dtype, g_dtype):
  """A contiguous gradient that is rounded anyway may start anywhere (a view into a larger buffer)."""
  from lewi_surge_b200 import ops
  dt = dict(bf16=torch.bfloat16, f32=torch.float32, f16=torch.float16)
  t, k, d = 37, 3, 64
  order = torch.randperm(t * k, device=cuda).to(torch.int32)
  pos = torch.empty_like(order)
  pos[order.long()] = torch.arange(t * k, dtype=torch.int32, device=cuda)
  y, w = torch.randn(t * k, d, device=cuda).to(dt[dtype]), torch.rand(t, k, device=cuda)
  g = torch.randn(t * d + 1, device=cuda).to(dt[g_dtype])[1:].view(t, d)
  assert g.is_contiguous() and g.data_ptr() % 16
  gy = g.to(y.dtype)
  dy, dw = ops.combine_bwd(y, pos.view(t, k), g, w, order)
  assert torch.equal(dy, ops.gather_rows(gy, order, w.reshape(-1), idx_div=k, scale_by_idx=True))
  assert torch.equal(dw, ops.gather_dot(y, pos.view(t, k), gy))
