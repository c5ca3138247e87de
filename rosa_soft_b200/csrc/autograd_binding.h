// Adds the differentiable operator to the extension module.
#pragma once

#include <torch/extension.h>

void bind_autograd(py::module_& m);
