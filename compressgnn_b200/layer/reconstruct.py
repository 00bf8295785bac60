"""Reconstruct node features from bucket representatives, fusing the shared bias and ReLU.

Drop-in for the reference's ``layer/CompressgnnReconstruct.py:11-42``:
``Compressgnn_Reconstruct(node_dim=-2).forward(src, index, bias=None, activation=None)``.
Unlike the reference, every CUDA call goes through the native gather (also without bias or
activation), and the bias gradient comes out of the same native call as the representative
gradient.
"""
import torch

from .. import runtime as _native


class _Reconstruct:
    """``apply(src, index, bias, relu, dropout_p=0.0)``: the native gather with its autograd node (in the
    binding).  A fresh dropout key per call comes from torch's host generator."""

    @staticmethod
    def apply(src, index, bias, relu, dropout_p=0.0):
        return _native.differentiable(_native.ops().reconstruct, src, index, bias, relu, dropout_p,
                                      _native.known_index_plan(index, src.size(0)))


class Compressgnn_Reconstruct(torch.nn.Module):
    def __init__(self, node_dim=-2):
        super().__init__()
        self.node_dim = node_dim

    def forward(self, src, index, bias=None, activation=None, dropout=0.0):
        """``dropout`` (not in the reference's signature): probability of the dropout that follows a ReLU
        activation, applied in the same pass; the caller passes 0 outside of training."""
        if activation not in (None, 'relu'):
            raise ValueError('Supported activations: None, relu')
        if dropout and activation != 'relu':
            raise ValueError('the fused dropout needs activation="relu"')
        if src.is_cuda and src.dim() == 2 and self.node_dim in (0, -2):
            return _Reconstruct.apply(src, index, bias, activation == 'relu', float(dropout))
        if src.is_cuda:
            output = src.index_select(self.node_dim, index)
            if bias is not None:
                output = output + bias
            output = output.relu() if activation == 'relu' else output
            return torch.nn.functional.dropout(output, dropout) if dropout else output
        raise RuntimeError("compressgnn_b200 runs on CUDA tensors only (no CPU reconstruct path)")
