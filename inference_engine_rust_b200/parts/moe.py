"""Mixture-of-experts feed-forward: `experts` small gated feed-forwards W_down (silu(W_gate h) * (W_up h)),
of which each token uses the `top` with the largest router logits z = W_r h + b (fp32), weighted by the
softmax over the chosen logits only; plus, optionally, a shared expert of the same form that every
token uses with weight 1.

Run as two products over all experts at once: the experts' gate and up matrices are stacked into one
[gate; up] matrix and their down matrices side by side, so that the activation row of a token is
[expert 0 | expert 1 | ... | shared]; the block of an expert the token did not choose is multiplied by
0 (by its routing weight otherwise) before the down product, which then sums exactly the chosen experts'
outputs and the shared one and adds them to the residual.  The products are the same projection kernels
the dense feed-forward uses, the step stays free of host decisions (CUDA graphs), and a token's result does
not depend on what the other tokens are; the price is that every expert's product is computed for every
token.  One-token steps and short prompts pay it gladly (all experts' weights are read anyway); longer prompts sort
their (token, choice) pairs by expert on the device and run each expert's products over its own rows alone
(`_forward_grouped`), the sums of a token's choices being added to the residual in order.  The step's number of tokens picks the form, and
the forms round differently: a prompt's result may differ in its last bits with how many tokens are batched beside it.

`GroupedMoE` (kind "grouped_moe") is the same with another router and another expert: scores are the softmax over ALL
router outputs, the choice is made on score + a stored `correction`, restricted to the `keep` best of `groups` equal
runs of neighbouring outputs (a run's score is its largest choice score), the weights are the chosen scores over
their sum; with `score: "sigmoid"` every output is scored by its own sigmoid instead, with `group_score: "top2_sum"` a
run's score is the sum of its two largest choice scores, and `route_scale` / `out_scale` multiply the weights; the last `identity` router outputs stand for experts without tensors that return their input; the
experts' activation is any member of the gated-activation family (`activation`, `limit`), and they have no
shared expert and no router bias.

`UngatedMoE` (kind "ungated_moe") takes the same router, with weights that may be the chosen scores as they are
(`renormalize: false`), and experts without a gate, W_down act(W_up h); a shared expert of the same form is multiplied by
sigmoid(W_sg h), one number per token.  The up product's epilogue applies the activation and each token's weight of the
expert that a column belongs to, so that nothing stands between the two products; W_sg is one more row of the router's
product, and the routing kernel adds the identity experts' share itself.
"""
from __future__ import annotations

from typing import Dict, Mapping

import torch

from ..config.specs import PartSpec
from ..csrc import bindings as B
from ..weights.loader import TensorSpec
from .base import FeedForward, Runtime, StepContext, register_part
from .linear import Linear


# Prompts of more than this many tokens compute a grouped router's logits (at most 32 outputs) with the kernel for few
# rows against a long matrix, the tokens being the matrix.
SKINNY_ROUTER_MIN_TOKENS = 32
# Up to this many tokens and router outputs the router's product and the routing are one kernel, a block per token whose eight warps take
# two outputs each.  More outputs are further rounds of them in every block, one kernel / two, us a mixture at a width of 4,096 with 8, 32 and 64
# tokens: 16 outputs 19.8 / 21.5, 30.4 / 37.1, 32.2 / 33.8; 32 outputs 24.8 / 22.2, 35.7 / 39.1, 39.2 / 37.2; 64 outputs 48 / 29, 68 / 51, 71 / 57; 128 outputs
# 98 / 54, 114 / 75, 114 / 82.
ROUTER_STEP_MAX_TOKENS = 64
ROUTER_STEP_MAX_OUTPUTS = 16
# Prompts of at least this many tokens run the experts' products over the tokens that chose them, if that is less than half of
# the rows that all experts over all tokens would have, and where two costs of the sorted form are outweighed:
#   a row's way through the sort, the gather and the sum: the experts left out must hold enough work, E F >= 2,048 top;
#   a row tile that an expert does not fill, above all where its width does not fill a tile's columns either: T F >= 48 K.
# Up to 2 M numbers in the sorted rows (T top H) both forms take their launches' time and the rows' way costs nothing.
# Grouped / all experts, us a mixture (T of 256, 384, 1,024, 2,048), E x F, chosen, width H:
#   16 x 768, 2, 4,096   112 / 139   115 / 162   136 / 247   168 / 447        8 x 1,792, 2, 4,096    98 / 117   101 / 156   146 / 285   234 / 525
#   16 x 896, 4, 4,096   126 / 146   119 / 172   170 / 289   289 / 531        64 x 512, 6, 2,048    136 / 145   136 / 186   160 / 343   230 / 617
#   32 x 384, 4, 4,096   108 / 121   111 / 132   137 / 251   220 / 457        128 x 256, 8, 2,048   145 / 144   152 / 186   188 / 345   266 / 621
#   256 x 64, 8, 4,096   245 / 154   264 / 209   327 / 345   418 / 618 (768 tokens 299 / 311: the second cost)
#   64 x 128, 8, 4,096   145 / 106   157 / 146   215 / 201   337 / 330        128 x 64, 8, 2,048    110 / 81    114 / 95    144 / 135   223 / 185 (the first)
# and at T of 384, 1,024, 4,096: 16 x 128, 4, 4,096   76 / 56   105 / 65   276 / 187        32 x 64, 8, 2,048    65 / 46   102 / 57   308 / 115
#   8 x 256, 2, 4,096    60 / 55   81 / 62   184 / 184                                      8 x 64, 2, 1,024     32 / 33   36 / 38    68 / 39
GROUPED_MIN_TOKENS = 384
GROUPED_ANY_NUMBERS = 2 << 20
GROUPED_MIN_LEFT_OUT = 2048
GROUPED_MIN_TILE_WORK = 48 << 10
# ... in equal portions of at most this many tokens, and of at most this many bytes for the sorted rows, their activations and their
# results: top x (4 H + 2 F) a token, 36 KB for two experts of 768 chosen at a width of 4,096 and 140 KB for eight of 512.  Every portion
# reads the experts' weights again: 8,192 tokens in portions of 8,192 / 4,096 / 2,048 take 522 / 540 / 659 us at the first of these sizes,
# 1,570 / 1,670 / 2,004 at the second.
GROUPED_MAX_TOKENS = 8192
GROUPED_MAX_BYTES = 512 << 20


class MoE(FeedForward):
    graph_safe = True

    def __init__(self, spec, rt: Runtime):
        self.rt = rt
        self.hidden_size = int(spec["hidden_size"])
        self.experts = int(spec["experts"])
        self.top = int(spec["top"])
        self.expert_ff = int(spec["expert_ff"])
        self.shared_ff = int(spec["shared_ff"]) if spec.get("shared_ff") else 0
        self.inter = self.experts * self.expert_ff + self.shared_ff
        self.act = B.gated_act(spec.get("activation", "silu"), spec.get("limit"))     # None: SiLU
        self.router = self.router_bias = self.gate_up = self.down = None

    def tensor_specs(self) -> Dict[str, TensorSpec]:
        h, f = self.hidden_size, self.expert_ff
        out = {"router": TensorSpec((self.experts, h)), "router.b": TensorSpec((self.experts,))}
        for e in range(self.experts):
            out[f"e{e}.gate"] = TensorSpec((f, h))
            out[f"e{e}.up"] = TensorSpec((f, h))
            out[f"e{e}.down"] = TensorSpec((h, f))
        if self.shared_ff:
            out["shared.gate"] = TensorSpec((self.shared_ff, h))
            out["shared.up"] = TensorSpec((self.shared_ff, h))
            out["shared.down"] = TensorSpec((h, self.shared_ff))
        return out

    def _load_experts(self, tensors: Mapping[str, torch.Tensor]) -> None:
        dt = self.rt.dtype
        names = [f"e{e}" for e in range(self.experts)] + (["shared"] if self.shared_ff else [])
        gate_up = torch.cat([tensors[f"{n}.gate"].to(dt) for n in names] + [tensors[f"{n}.up"].to(dt) for n in names], dim=0)
        self.gate_up = Linear(gate_up, self.rt)
        self.down = Linear(torch.cat([tensors[f"{n}.down"].to(dt) for n in names], dim=1), self.rt)
        self.router = Linear(tensors["router"], self.rt)

    def load(self, tensors: Mapping[str, torch.Tensor]) -> None:
        self._load_experts(tensors)
        self.router_bias = tensors["router.b"].to(torch.float32).contiguous()

    def weight_bytes(self) -> int:
        return self.gate_up.nbytes() + self.down.nbytes() + self.router.nbytes()

    def _router_logits(self, xn, N: int, T: int, stream: int):
        """The fp32 product of the step's rows with the router's N rows, and whether it lies by output ([N, T]) or by token."""
        ws = self.rt.workspace
        by_output = False
        if (self.rt.fast and T > SKINNY_ROUTER_MIN_TOKENS and N <= 32 and isinstance(xn, torch.Tensor)
                and xn.dtype == torch.bfloat16 and self.router.weight.dtype == torch.bfloat16):
            # A prompt: few router outputs against many tokens.  A token tile of the tensor-core product would carry
            # N columns and 128-token tiles alone leave most of the device idle; the kernel for few rows against a long
            # matrix takes the router's rows as its "tokens" and the tokens as the matrix it streams, 16 tokens per
            # CTA, and leaves the logits with a row per router output.
            z = ws.take("moe.logits_by_output", (N, T), torch.float32)
            # the streamed "matrix" is the step's rows, which the norm in front has just written
            by_output = B.gemm_rows(self.router.weight, xn[:T], z, N, B.GEMM_STORE, self.rt.err, stream, w_dynamic=True)
        if not by_output:
            z = ws.take("moe.logits", (T, N), torch.float32)
            self.router.apply(xn, z, T, stream)
        return z, by_output

    def _routes_in_one(self, xn, T: int) -> bool:
        """Steps of few tokens over few outputs: one kernel for the router's product and the routing."""
        return (self.rt.fast and T <= ROUTER_STEP_MAX_TOKENS and self.router.out_features <= ROUTER_STEP_MAX_OUTPUTS
                and isinstance(xn, torch.Tensor) and xn.dtype == torch.bfloat16)

    def _route(self, xn, residual, T: int, stream: int):
        """(wt [T, E or more] dense routing weights, idx, w [T, top] the choices); the share of experts that return their
        input is added to `residual`."""
        ws, E = self.rt.workspace, self.experts
        wt = ws.take("moe.weights", (T, E + (1 if self.shared_ff else 0)), torch.float32)
        idx = ws.take("moe.chosen", (T, self.top), torch.int32)
        w = ws.take("moe.chosen_weights", (T, self.top), torch.float32)
        if self._routes_in_one(xn, T) and B.router_step(xn, self.router.weight, T, E, self.top, wt, idx, w, stream, bias=self.router_bias):
            return wt, idx, w
        z, by_output = self._router_logits(xn, E, T, stream)
        B.router_topk(z, self.router_bias, T, E, self.top, wt, idx, w, stream, by_output=by_output)
        return wt, idx, w

    def _portion(self) -> int:
        """Tokens of a grouped portion at most."""
        return min(GROUPED_MAX_TOKENS, GROUPED_MAX_BYTES // (self.top * (4 * self.hidden_size + 2 * self.expert_ff)))

    def _takes_grouped(self, xn, T: int, residual=None) -> bool:
        E, F, H = self.experts, self.expert_ff, self.hidden_size
        return (self.rt.fast and min(T, self._portion()) >= GROUPED_MIN_TOKENS and T * E >= 2 * (T * self.top + 64 * E) and E <= 1024
                and (T * self.top * H <= GROUPED_ANY_NUMBERS
                     or (E * F >= GROUPED_MIN_LEFT_OUT * self.top and T * F >= GROUPED_MIN_TILE_WORK))
                and isinstance(xn, torch.Tensor) and xn.dtype == torch.bfloat16 and xn.stride(0) % 8 == 0
                and xn.data_ptr() % 16 == 0 and F % 64 == 0 and H % 8 == 0 and self.shared_ff % 8 == 0
                # (a token's results are added to its residual by 16-byte accesses)
                and (residual is None or (residual.stride(0) % 4 == 0 and residual.data_ptr() % 16 == 0)))

    def _forward_grouped(self, xn, residual, T: int, stream: int) -> None:
        """One portion of a prompt: the choices sorted by expert, each expert's products over its own rows, the shared expert
        over all rows, then a token's results added to its residual."""
        rt, ws, E, F, H, top, S = self.rt, self.rt.workspace, self.experts, self.expert_ff, self.hidden_size, self.top, self.shared_ff
        _, idx, w = self._route(xn, residual, T, stream)
        rows, tiles = T * top, T * top // 128 + E
        groups = ws.take("moe.groups", (B.moe_group_ints(T, top, E),), torch.int32)
        pos = ws.take("moe.pos", (rows,), torch.int32)
        row_token = ws.take("moe.row_token", (rows,), torch.int32)
        row_w = ws.take("moe.row_weight", (rows,), torch.float32)
        B.moe_sort(idx, w, T, top, E, groups, pos, row_token, row_w, stream)
        y = ws.take("moe.results", (rows, H), torch.float32)
        xs = y.view(torch.bfloat16).flatten()[:rows * H].view(rows, H)       # the sorted rows are done with when their results are written
        B.moe_gather(xn, groups, row_token, rows, xs, stream)
        act = ws.take("moe.act", (rows, F), torch.bfloat16)
        B.gemm_tc_grouped_gated(xs, self.gate_up.weight, act, groups, tiles, E, F, self.inter, row_w, rt.err, stream, fn=self.act)
        B.gemm_tc_grouped(act, self.down.weight, y, groups, tiles, E, F, rt.err, stream)
        if S:
            act_s = ws.take("ffn.act", (T, S), torch.bfloat16)
            if not (B.gemm_tc_gated(xn, self.gate_up.weight[E * F:], act_s, T, rt.err, stream, fn=self.act, inter=S, up_rows=self.inter)
                    and B.gemm_tc(act_s, self.down.weight[:, E * F:], residual, T, B.GEMM_ADD_RESIDUAL, rt.err, stream)):
                raise B.KernelError("grouped experts: the shared expert's products were refused")
        B.moe_combine(y, pos, w, T, top, residual, stream)

    def forward(self, xn, residual, ctx: StepContext) -> None:
        rt, ws, T, I, E = self.rt, self.rt.workspace, ctx.n_tokens, self.inter, self.experts
        if self._takes_grouped(xn, T, residual):
            size = -(-T // -(-T // self._portion()))
            for t in range(0, T, size):
                n = min(size, T - t)
                self._forward_grouped(xn[t:t + n], residual[t:t + n], n, ctx.stream)
            return
        wt, _, _ = self._route(xn, residual, T, ctx.stream)
        act = ws.take("ffn.act", (T, I), rt.dtype)
        done = False
        if rt.fast:
            from . import fast_linear
            # every block of columns times its expert's weight, in the product's own kernel
            factor = B.epilogue(scale=wt, blocks=wt.shape[1] - 1, block_cols=self.expert_ff)
            done = fast_linear.apply_gated(self.gate_up, xn, act, T, ctx.stream, fn=self.act, epilogue=factor)
        if not done:
            gu = ws.take("ffn.gate_up", (T, 2 * I), rt.dtype)
            self.gate_up.apply(xn, gu, T, ctx.stream)
            if self.act is None:
                B.silu_mul(gu, act, T, I, ctx.stream)
            else:
                B.gated_act_mul(gu, act, T, I, self.act, ctx.stream)
            B.moe_scale(act, wt, T, E, self.expert_ff, ctx.stream)
        self.down.apply(act, residual, T, ctx.stream, add_residual=True, ctx=ctx)


class GroupedMoE(MoE):
    graph_safe = True
    takes_out_scale = True

    def __init__(self, spec, rt: Runtime):
        super().__init__(spec, rt)
        self.identity = int(spec.get("identity") or 0)
        self.outputs = self.experts + self.identity
        self.groups = int(spec.get("groups") or 1)
        self.keep = int(spec.get("keep") or self.groups)
        self.score = spec.get("score") or "softmax"
        self.group_score = spec.get("group_score") or "max"
        if self.score not in B.ROUTER_SCORES or self.group_score not in B.ROUTER_GROUP_SCORES:
            raise ValueError(f"grouped_moe: score must be one of {sorted(B.ROUTER_SCORES)} and group_score one of "
                             f"{sorted(B.ROUTER_GROUP_SCORES)}, got {self.score!r} and {self.group_score!r}")
        self.weight_eps = float(spec.get("weight_eps", 1e-20))
        # both factors multiply the routing weights (fp32), in which the feed-forward's result is linear
        self.weight_scale = float(spec.get("route_scale", 1.0)) * float(spec.get("out_scale", 1.0))
        if self.shared_ff:
            raise ValueError("grouped_moe has no shared expert")
        if self.outputs % self.groups:
            raise ValueError(f"{self.outputs} router outputs do not form {self.groups} equal groups")
        if not 0 < self.keep <= self.groups or self.top > self.keep * (self.outputs // self.groups):
            raise ValueError(f"top {self.top} does not fit into {self.keep} of {self.groups} groups of "
                             f"{self.outputs // self.groups}")
        self.correction = None

    def tensor_specs(self) -> Dict[str, TensorSpec]:
        out = super().tensor_specs()
        del out["router.b"]
        out["router"] = TensorSpec((self.outputs, self.hidden_size))
        out["correction"] = TensorSpec((self.outputs,))
        return out

    def load(self, tensors: Mapping[str, torch.Tensor]) -> None:
        self._load_experts(tensors)
        self.correction = tensors["correction"].to(torch.float32).contiguous()

    def _route(self, xn, residual, T: int, stream: int):
        ws, E, N = self.rt.workspace, self.experts, self.outputs
        wt = ws.take("moe.weights", (T, E), torch.float32)
        wid = ws.take("moe.identity_share", (T,), torch.float32)
        idx = ws.take("moe.chosen", (T, self.top), torch.int32)
        w = ws.take("moe.chosen_weights", (T, self.top), torch.float32)
        if self._routes_in_one(xn, T) and B.router_step(
                xn, self.router.weight, T, E, self.top, wt, idx, w, stream, N=N, wid=wid, residual=residual if self.identity else None,
                grouped=dict(correction=self.correction, groups=self.groups, keep=self.keep, score=self.score, group_score=self.group_score,
                             weight_eps=self.weight_eps, weight_scale=self.weight_scale)):
            return wt, idx, w
        z, by_output = self._router_logits(xn, N, T, stream)
        B.router_grouped(z, self.correction, T, E, N, self.top, self.groups, self.keep, wt, wid, idx, w, stream,
                         by_output=by_output, score=self.score, group_score=self.group_score, weight_eps=self.weight_eps,
                         weight_scale=self.weight_scale, x=xn if self.identity else None, residual=residual if self.identity else None)
        return wt, idx, w


class UngatedMoE(GroupedMoE):
    graph_safe = True

    def __init__(self, spec, rt: Runtime):
        shared = int(spec["shared_ff"]) if spec.get("shared_ff") else 0
        super().__init__(PartSpec(spec.kind, {**spec.params, "shared_ff": None, "activation": "silu"}), rt)
        self.shared_ff = shared
        self.inter = self.experts * self.expert_ff + shared
        self.activation = spec.get("activation", "gelu")
        self.renormalize = bool(spec.get("renormalize", True))
        self.router_rows = self.outputs + (1 if shared else 0)
        self.wt_cols = self.experts + (1 if shared else 0)
        self.up = None

    def tensor_specs(self) -> Dict[str, TensorSpec]:
        h, f, s = self.hidden_size, self.expert_ff, self.shared_ff
        out = {"router": TensorSpec((self.outputs, h)), "correction": TensorSpec((self.outputs,))}
        for e in range(self.experts):
            out[f"e{e}.up"], out[f"e{e}.down"] = TensorSpec((f, h)), TensorSpec((h, f))
        if s:
            out["shared.up"], out["shared.down"], out["shared.sg"] = TensorSpec((s, h)), TensorSpec((h, s)), TensorSpec((1, h))
        return out

    def load(self, tensors: Mapping[str, torch.Tensor]) -> None:
        dt = self.rt.dtype
        names = [f"e{e}" for e in range(self.experts)] + (["shared"] if self.shared_ff else [])
        self.up = Linear(torch.cat([tensors[f"{n}.up"].to(dt) for n in names], dim=0), self.rt)
        self.down = Linear(torch.cat([tensors[f"{n}.down"].to(dt) for n in names], dim=1), self.rt)
        rows = [tensors["router"].to(dt)] + ([tensors["shared.sg"].to(dt)] if self.shared_ff else [])
        self.router = Linear(torch.cat(rows, dim=0), self.rt)
        self.correction = tensors["correction"].to(torch.float32).contiguous()

    def weight_bytes(self) -> int:
        return self.up.nbytes() + self.down.nbytes() + self.router.nbytes()

    def forward(self, xn, residual, ctx: StepContext) -> None:
        rt, ws, T, E = self.rt, self.rt.workspace, ctx.n_tokens, self.experts
        z, by_output = self._router_logits(xn, self.router_rows, T, ctx.stream)
        wt = ws.take("moe.weights", (T, self.wt_cols), torch.float32)
        wid = ws.take("moe.identity_share", (T,), torch.float32)
        idx = ws.take("moe.chosen", (T, self.top), torch.int32)
        w = ws.take("moe.chosen_weights", (T, self.top), torch.float32)
        B.router_grouped(z, self.correction, T, E, self.outputs, self.top, self.groups, self.keep, wt, wid, idx, w, ctx.stream,
                         by_output=by_output, score=self.score, group_score=self.group_score, weight_eps=self.weight_eps,
                         weight_scale=self.weight_scale, renormalize=self.renormalize, shared_gate=bool(self.shared_ff),
                         x=xn if self.identity else None, residual=residual if self.identity else None)
        act = ws.take("ffn.act", (T, self.inter), rt.dtype)
        self.up.apply(xn, act, T, ctx.stream, epilogue=B.epilogue(self.activation, scale=wt, blocks=E if self.shared_ff else E - 1,
                                                                  block_cols=self.expert_ff))
        self.down.apply(act, residual, T, ctx.stream, add_residual=True, ctx=ctx)


register_part("ffn", "ungated_moe", UngatedMoE)
register_part("ffn", "moe", MoE)
register_part("ffn", "grouped_moe", GroupedMoE)
