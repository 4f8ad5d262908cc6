// Python bindings of the native host side.
#include <torch/extension.h>

#include "host.h"

namespace py = pybind11;
using namespace st_host;

namespace {
using Release = py::call_guard<py::gil_scoped_release>;
py::object maybe(const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); }
py::tuple plan_tensors(const Plan& p) { return py::make_tuple(maybe(p.order_tensor()), maybe(p.tmap_tensor()), maybe(p.tmask_tensor())); }
}  // namespace

PYBIND11_MODULE(_st_host, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const TypeError& e) {
      PyErr_SetString(PyExc_TypeError, e.what());
    } catch (const ValueError& e) {
      PyErr_SetString(PyExc_ValueError, e.what());
    }
  });
  py::class_<MapState, MapPtr>(m, "MapState")
      .def(py::init([]() { return c10::make_intrusive<MapState>(); }))
      .def("plan", [](MapState& s, const Tensor& nbr, bool row_order) { return plan_tensors(s.plan(nbr, row_order)); })
      .def("inverse_plan", [](MapState& s, const Tensor& nbr, int64_t n_in, bool row_order) -> py::object {
        const Plan* p = s.inverse_plan(nbr, n_in, row_order);
        return p ? py::object(plan_tensors(*p)) : py::none();
      })
      .def("inverse", &MapState::inverse, Release())
      .def("inverse_state", &MapState::inverse_state, Release())
      .def("symmetric", &MapState::symmetric, Release())
      .def("pairs", &MapState::pairs, Release());
  py::class_<OutCoords, c10::intrusive_ptr<OutCoords>>(m, "OutCoords")
      .def(py::init([](const Tensor& coords, int k, int s, int d, int p, bool transposed, std::vector<int64_t> new_shape,
                       std::vector<int64_t> in_shape, int64_t batch_bound, bool with_map) {
        return c10::make_intrusive<OutCoords>(coords, k, s, d, p, transposed, new_shape, in_shape, batch_bound, with_map);
      }))
      .def("finish", [](OutCoords& o) {
        std::tuple<Tensor, Tensor, c10::optional<MapPtr>> r;
        {
          py::gil_scoped_release release;
          r = o.finish();
        }
        const auto& map = std::get<2>(r);
        return py::make_tuple(std::get<0>(r), maybe(std::get<1>(r)), map ? py::cast(*map) : py::none());
      });
  m.def("submanifold", [](const Tensor& coords, std::vector<int64_t> shape, int k, int d, double factor,
                          const c10::optional<Tensor>& keys, const c10::optional<Tensor>& vals) {
    std::tuple<Tensor, Tensor, Tensor, Tensor, MapPtr> r;
    {
      py::gil_scoped_release release;
      r = submanifold(coords, std::move(shape), k, d, factor, keys, vals);
    }
    return py::make_tuple(std::get<0>(r), std::get<1>(r), maybe(std::get<2>(r)), std::get<3>(r), std::get<4>(r));
  });
  m.def("probe_map", &probe_map, Release());
  m.def("build_table", &build_table, Release());
  m.def("extent", &extent, Release());
  m.def("conv", &conv, Release());
  m.def("conv_hashfly", &conv_hashfly, Release());
  m.def("conv_forward", &conv_forward, Release());
  m.def("conv_dgrad", &conv_dgrad, Release());
  m.def("conv_wgrad", [](const Tensor& x, const Tensor& dy, const Tensor& nbr, const MapPtr& map, bool row_order) {
    return conv_wgrad(x, dy, nbr, map, x.scalar_type(), row_order);
  }, Release());
  m.def("batch_info", &batch_info, Release());
  m.def("batch_norm_train", &batch_norm_train, Release());
  m.def("batch_norm_running", &batch_norm_running, Release());
  m.def("concat_cols", &concat_cols, Release());
  m.def("pool", &pool, Release());
  m.def("to_dense", &to_dense, Release());
  m.def("trace_start", &trace_start);
  m.def("trace_stop", &trace_stop);
  m.def("trace_spans", &trace_spans, Release());
}
